"""Performance cases: the calls that a user of gbpowspec has on the GPU, over the sizes they come in.

Every case goes through a public entry point:

    pk       PowerSpectrum.run         resident pipeline, one mock (what power_multipoles runs)
    batch    BatchRunner.run           many uneven mocks of one mesh through resident lanes
    deposit  cic_mas_vec               the reference's mass assignment (drop-in)
    powspec  powspec_vec               the reference's P_l(k) of a mesh (drop-in)
    xi       xi_vec                    the reference's xi_l(r) of a mesh (drop-in)
    bispec   bispec                    the reference's bispectrum of a mesh (drop-in)
    grad     power_multipoles_diff     P_l(k) and its gradients, a step of a fit to a spectrum

Catalogues are half uniform, half clumped (Gaussian clumps of about 32 particles, 4 Mpc/h) with a
redshift-space shift along z; meshes are lognormal contrasts.  P_l is kept as float32, the type the
reference's powspec_vec returns it in and the precision of the estimator's own arithmetic.
"""
import math
import sys

import numpy as np
import torch

sys.path.insert(0, "jax-powspec_gb300")      # the package lives in this folder of the repository

MAS = {"ngp": 1, "cic": 2, "tsc": 3, "pcs": 4}
ELL_FACTORS = (1.0, 5.0, 9.0)


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one call on a small catalogue: what a sampler or a quick look pays per evaluation
        {"name": "pk_64_cic", "kind": "pk", "mesh": 64, "n": 20011, "mas": "cic", "interlace": False,
         "weights": False, "box": 400.0, "ells": "02", "bins": "unit"},
        # an ordinary survey-like catalogue: weighted tracers
        {"name": "pk_256_tsc_weighted", "kind": "pk", "mesh": 256, "n": 1000003, "mas": "tsc", "interlace": True,
         "weights": True, "box": 1000.0, "ells": "024", "bins": "unit"},
        # the headline workload: 4 Mi particles, 512^3, TSC + interlacing
        {"name": "pk_512_tsc", "kind": "pk", "mesh": 512, "n": 4194304, "mas": "tsc", "interlace": True,
         "weights": False, "box": 2500.0, "ells": "024", "bins": "unit"},
        # the largest configuration: 16 Mi particles, 1024^3, PCS + interlacing
        {"name": "pk_1024_pcs", "kind": "pk", "mesh": 1024, "n": 16777216, "mas": "pcs", "interlace": True,
         "weights": False, "box": 2000.0, "ells": "024", "bins": "unit"},
        # a mesh side chosen for its cell size, not a power of two
        {"name": "pk_360_cic", "kind": "pk", "mesh": 360, "n": 1500007, "mas": "cic", "interlace": True,
         "weights": False, "box": 1800.0, "ells": "02", "bins": "unit"},
        # a covariance set: uneven mocks of one mesh through the lanes
        {"name": "batch_128_cic", "kind": "batch", "mesh": 128, "mocks": 24, "n_min": 200000, "n_max": 2000000,
         "mas": "cic", "interlace": True, "box": 1500.0, "ells": "02"},
        # the reference's own first step at its smaller and its headline size
        {"name": "deposit_128", "kind": "deposit", "mesh": 128, "n": 1048576, "box": 1000.0},
        {"name": "deposit_512", "kind": "deposit", "mesh": 512, "n": 4194304, "box": 2500.0},
        # the reference's own second step
        {"name": "powspec_512", "kind": "powspec", "mesh": 512, "box": 2500.0, "bins": "unit"},
        # the two-point function of a mesh, 50 separation shells
        {"name": "xi_256", "kind": "xi", "mesh": 256, "box": 1000.0, "s_max": 200.0, "ds": 4.0},
        # the bispectrum at k1 = 0.1, k2 = 0.2, 20 angles (the reference's own test case)
        {"name": "bispec_256", "kind": "bispec", "mesh": 256, "box": 2500.0, "k1": 0.1, "k2": 0.2, "angles": 20},
        # one step of a fit of positions and weights to a target monopole
        {"name": "grad_256_tsc", "kind": "grad", "mesh": 256, "n": 1048576, "mas": "tsc", "interlace": True,
         "weights": True, "box": 1000.0},
    ]


def _log_uniform(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def _mesh_side(rng, largest):
    """A power of two in most programs, any side in the others."""
    if rng.random() < 0.7:
        return rng.choice([s for s in (64, 128, 256, 512) if s <= largest])
    return int(_log_uniform(rng, 48, min(largest, 400)))


def _particles(rng, mesh):
    return int(_log_uniform(rng, 1e4, max(2e4, min(1e7, 5.0 * mesh ** 3))))


def draw(rng):
    kind = rng.choice(["pk", "pk", "pk", "pk", "batch", "deposit", "powspec", "powspec", "xi", "bispec", "grad"])
    box = round(rng.uniform(400.0, 3000.0), 1)
    if kind == "batch":
        mesh = rng.choice([64, 128, 256])
        n_max = _particles(rng, mesh)
        return {"kind": kind, "mesh": mesh, "mocks": rng.randint(3, 24), "n_min": max(1000, n_max // 10), "n_max": n_max,
                "mas": rng.choice(["cic", "tsc"]), "interlace": rng.random() < 0.7, "box": box,
                "ells": rng.choice(["02", "024"])}
    if kind == "pk":
        mesh = _mesh_side(rng, 512)
        return {"kind": kind, "mesh": mesh, "n": _particles(rng, mesh), "mas": rng.choice(["ngp", "cic", "tsc", "pcs"]),
                "interlace": rng.random() < 0.6, "weights": rng.random() < 0.3, "box": box,
                "ells": rng.choice(["0", "02", "024"]), "bins": rng.choice(["unit", "unit", "coarse", "corner"])}
    if kind == "deposit":
        mesh = _mesh_side(rng, 512)
        return {"kind": kind, "mesh": mesh, "n": _particles(rng, mesh), "box": box}
    if kind == "powspec":
        return {"kind": kind, "mesh": _mesh_side(rng, 512), "box": box, "bins": rng.choice(["unit", "coarse", "corner"])}
    mesh = _mesh_side(rng, 256)
    if kind == "xi":
        return {"kind": kind, "mesh": mesh, "box": box, "s_max": round(box * rng.uniform(0.1, 0.45), 1),
                "ds": round(box / mesh * rng.uniform(1.0, 4.0), 2)}
    if kind == "bispec":
        kf = 2.0 * math.pi / box
        mesh -= mesh % 4
        k1 = kf * rng.uniform(4.0, mesh / 10.0)
        return {"kind": kind, "mesh": mesh, "box": box, "k1": round(k1, 5), "k2": round(k1 * rng.uniform(1.0, 2.0), 5),
                "angles": rng.randint(5, 30)}
    mesh -= mesh % 2
    return {"kind": kind, "mesh": mesh, "n": min(2000000, _particles(rng, mesh)), "mas": rng.choice(["cic", "tsc", "pcs"]),
            "interlace": rng.random() < 0.5, "weights": rng.random() < 0.5, "box": box}


# ---------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _catalogue(n, box, gen, weights=False):
    """(x, y, z, w or None): float32, positions in [0, box)."""
    centres = torch.rand((3, max(1, n // 64)), generator=gen, device="cuda") * box
    host = torch.randint(centres.shape[1], (n,), generator=gen, device="cuda")
    clumped = torch.rand(n, generator=gen, device="cuda") < 0.5
    out = []
    for a in range(3):
        c = torch.where(clumped, centres[a][host] + 4.0 * torch.randn(n, generator=gen, device="cuda"),
                        box * torch.rand(n, generator=gen, device="cuda"))
        if a == 2:
            c = c + 3.0 * torch.randn(n, generator=gen, device="cuda")
        c = torch.remainder(c, box)
        out.append(torch.clamp(c, max=float(np.nextafter(np.float32(box), np.float32(0)))).contiguous())
    w = 0.5 + torch.rand(n, generator=gen, device="cuda") if weights else None
    return out[0], out[1], out[2], w


def _contrast(mesh, box, gen):
    """A lognormal density contrast, float32 [mesh]^3, mean 0."""
    g = torch.fft.rfftn(torch.randn((mesh, mesh, mesh), generator=gen, device="cuda"))
    k = [2.0 * math.pi / box * torch.fft.fftfreq(mesh, 1.0 / mesh, device="cuda") for _ in range(2)]
    k.append(2.0 * math.pi / box * torch.fft.rfftfreq(mesh, 1.0 / mesh, device="cuda"))
    kk = (k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2).sqrt()
    g = torch.fft.irfftn(g * (kk * torch.exp(-(kk / 0.3) ** 2)).sqrt(), s=(mesh, mesh, mesh))
    rho = torch.exp(0.8 * g / g.std())
    return (rho / rho.mean() - 1.0).contiguous()


def _edges_kf(case):
    """k edges in units of the fundamental frequency, float32."""
    h = case["mesh"] // 2
    if case["bins"] == "coarse":                 # a data vector: three modes wide, up to half the Nyquist frequency
        return np.arange(1.0, max(5.0, 0.5 * h), 3.0).astype(np.float32)
    if case["bins"] == "corner":                 # every mode, the corners of the cube among them
        return np.arange(1.0, math.sqrt(3.0) * h + 2.0, 1.0).astype(np.float32)
    return np.arange(1, h).astype(np.float32)    # kF .. k_Nyquist, one kF wide


def _counts(case):
    m = case["mocks"]
    r = [case["n_min"] * (case["n_max"] / case["n_min"]) ** (((7 * i) % m) / max(1, m - 1)) for i in range(m)]
    return [min(case["n_max"], int(v)) for v in r]


def _ells(case):
    return tuple(int(c) for c in case["ells"])


def _k_edges(case):
    kf = np.float32(np.float32(2.0 * np.pi) / np.float32(case["box"]))
    return (_edges_kf(case) * kf).astype(np.float32)


def _s_edges(case):
    return np.arange(case["ds"], case["s_max"], case["ds"]).astype(np.float32)


def _theta(case):
    return np.linspace(0.05, math.pi - 0.05, case["angles"]).astype(np.float32)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    st = {"case": case}
    if kind == "pk":
        from gbpowspec import PkConfig, PowerSpectrum
        cfg = PkConfig(n_mesh=case["mesh"], box_size=case["box"], mas=case["mas"], interlace=case["interlace"],
                       ells=_ells(case), k_edges_kf=tuple(_edges_kf(case).tolist()))
        st["plan"] = PowerSpectrum(cfg)
        st["plan"].reserve(case["n"])
        st["xyzw"] = _catalogue(case["n"], case["box"], gen, case["weights"])
    elif kind == "batch":
        from gbpowspec.batch import BatchRunner, ParticleArena
        counts = _counts(case)
        arena = ParticleArena.empty(counts)
        for i, n in enumerate(counts):
            for view, c in zip(arena.views(i), _catalogue(n, case["box"], gen)):
                view.copy_(c)
        st["runner"] = BatchRunner(case["mesh"], capacity=case["n_max"], mas=case["mas"], interlace=case["interlace"],
                                   ells=_ells(case), n_lanes=3, tiles=None)
        st["arena"] = arena
        st["jobs"] = arena.job_table(case["box"], case["mesh"])
        st["out"] = st["runner"].alloc_result(len(counts))
    elif kind == "deposit":
        st["xyzw"] = _catalogue(case["n"], case["box"], gen)
        st["w"] = torch.ones(case["n"], device="cuda")
        st["delta"] = torch.zeros((case["mesh"],) * 3, device="cuda")
    elif kind in ("powspec", "xi", "bispec"):
        st["delta"] = _contrast(case["mesh"], case["box"], gen)
        if kind == "powspec":
            st["k_edges"] = _k_edges(case)
        elif kind == "xi":
            st["s_edges"] = _s_edges(case)
        else:
            st["theta"] = _theta(case)
    else:
        x, y, z, w = _catalogue(case["n"], case["box"], gen, case["weights"])
        st["leaves"] = [t.requires_grad_(True) for t in (x, y, z, w) if t is not None]
        st["target"] = _target(case)
    return st


def _target(case):
    """The monopole that a fit aims at, one value per default bin (kF .. k_Nyquist in steps of kF), float64."""
    kf = 2.0 * math.pi / case["box"]
    k = np.arange(kf, math.pi * case["mesh"] / case["box"], kf).astype(np.float32)
    k = torch.from_numpy(0.5 * (k[1:].astype(np.float64) + k[:-1])).cuda()
    return 3.0 * case["box"] ** 3 / case["n"] * (1.0 + 1.0 / (0.01 + k))


def _fit_grads(pk, target, leaves):
    loss = ((pk[:, 0] - target) / target).square().mean()
    return torch.autograd.grad(loss, leaves)


# ---------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "pk":
        r = st["plan"].run(*st["xyzw"])
        return {"pk": r.pk.float(), "k_mean": r.k_mean, "nmodes": r.nmodes}
    if kind == "batch":
        r = st["runner"].run(st["jobs"], st["out"])
        return {"pk": r.pk.float(), "k_mean": r.kmean, "nmodes": r.nmodes}
    if kind == "deposit":
        from gbpowspec import cic_mas_vec
        x, y, z, _ = st["xyzw"]
        return cic_mas_vec(st["delta"], x, y, z, st["w"], case["n"], 0.0, 0.0, 0.0, case["box"], case["mesh"], True)
    if kind == "powspec":
        from gbpowspec import powspec_vec
        return powspec_vec(st["delta"], case["box"], st["k_edges"])
    if kind == "xi":
        from gbpowspec import xi_vec
        return xi_vec(st["delta"], case["box"], st["s_edges"])
    if kind == "bispec":
        from gbpowspec import bispec
        return bispec(st["delta"], case["box"], case["k1"], case["k2"], st["theta"])
    from gbpowspec import power_multipoles_diff
    pk = power_multipoles_diff(*st["leaves"], box_size=case["box"], n_mesh=case["mesh"], mas=case["mas"],
                               interlace=case["interlace"])
    return {"pk": pk.detach().float(), "grads": _fit_grads(pk, st["target"], st["leaves"])}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Inputs read once, outputs written once; the transforms' and the deposits' operations."""
    kind, N = case["kind"], case["mesh"]
    M = N ** 3
    fft = 2.5 * M * math.log2(M)                                     # one real transform
    if kind in ("pk", "grad"):
        g = 2 if case["interlace"] else 1
        per = 16 if case["weights"] else 12
        dep = 2.0 * case["n"] * g * MAS[case["mas"]] ** 3
        if kind == "pk":
            return {"bytes": case["n"] * per + len(_edges_kf(case)) * 28, "flops": g * (fft + 4.0 * M) + dep}
        return {"bytes": 2 * case["n"] * per + N * 12, "flops": g * (2 * fft + 10.0 * M) + 5 * dep}
    if kind == "batch":
        g = 2 if case["interlace"] else 1
        n = sum(_counts(case))
        return {"bytes": 12 * n + case["mocks"] * N * 20,
                "flops": case["mocks"] * g * (fft + 4.0 * M) + 2.0 * n * g * MAS[case["mas"]] ** 3}
    if kind == "deposit":
        return {"bytes": 16 * case["n"] + 8 * M, "flops": 16.0 * case["n"]}
    if kind == "powspec":
        return {"bytes": 4 * M + len(_edges_kf(case)) * 20, "flops": fft + 4.0 * M}
    if kind == "xi":
        return {"bytes": 4 * M + len(_s_edges(case)) * 20, "flops": 2 * fft + 10.0 * M}
    return {"bytes": 4 * M + case["angles"] * 20, "flops": 7 * fft + 12.0 * M}


# ---------------------------------------------------------------- the same in 64 bits (plain torch)
def _signed(N):
    i = torch.arange(N, device="cuda")
    return torch.where(i > N // 2, i - N, i)


def _bin_of_k2(edges, top):
    """Bin of every integer k^2 <= top (-1: none): float32 |k| against the float32 edges, the last one closed."""
    e = torch.from_numpy(np.asarray(edges, np.float32)).cuda()
    k = torch.arange(top + 1, device="cuda").to(torch.float32).sqrt()
    b = torch.searchsorted(e, k, right=True) - 1
    b = torch.where(k == e[-1], torch.full_like(b, e.numel() - 2), b)
    return torch.where(b < e.numel() - 1, b, torch.full_like(b, -1))


def _legendre_sums(power, kz, N, edges, out=None):
    """[nb, 3] sums of power x L_0,2,4(mu) and [nb] mode counts; power(x0, x1) gives planes x0..x1 over (ky, kz)."""
    h = N // 2
    top = 3 * h * h
    tot = torch.zeros((4, top + 1), dtype=torch.float64, device="cuda")
    ki = _signed(N)
    step = max(1, min(N, (1 << 26) // (N * kz.numel())))
    for x0 in range(0, N, step):
        k2 = (ki[x0:x0 + step, None, None] ** 2 + ki[None, :, None] ** 2 + kz[None, None, :] ** 2)
        mu2 = (kz[None, None, :] ** 2).double() / k2.clamp(min=1).double()
        p = power(x0, min(N, x0 + step))
        flat = k2.reshape(-1)
        for q in range(3):
            tot[q] += torch.bincount(flat, weights=(p * mu2 ** q).reshape(-1), minlength=top + 1)
        tot[3] += torch.bincount(flat, minlength=top + 1)
    b = _bin_of_k2(edges, top)
    keep = b >= 0
    nb = len(edges) - 1
    m = torch.zeros((4, nb), dtype=torch.float64, device="cuda").index_add_(1, b[keep], tot[:, keep])
    sums = torch.stack([m[0], 1.5 * m[1] - 0.5 * m[0], (35 * m[2] - 30 * m[1] + 3 * m[0]) / 8], dim=1)
    k = torch.arange(top + 1, device="cuda").double().sqrt()
    ksum = torch.zeros(nb, dtype=torch.float64, device="cuda").index_add_(0, b[keep], (k * tot[3])[keep])
    return sums, m[3], ksum


def _bspline(u, mas, half):
    u = u + 0.5 if half else u
    i = torch.floor(u)
    d = u - i
    i = i.long()
    if mas == 1:
        return i + (d >= 0.5).long(), [torch.ones_like(d)]
    if mas == 2:
        return i, [1.0 - d, d]
    if mas == 3:
        up = d >= 0.5
        s = torch.where(up, d - 1.0, d)
        return i + up.long() - 1, [0.5 * (0.5 - s) ** 2, 0.75 - s * s, 0.5 * (0.5 + s) ** 2]
    m = 1.0 - d
    return i - 1, [m ** 3 / 6, (4 - 6 * d * d + 3 * d ** 3) / 6, (4 - 6 * m * m + 3 * m ** 3) / 6, d ** 3 / 6]


def _mesh64(us, w, N, mas, half):
    (fx, wx), (fy, wy), (fz, wz) = (_bspline(u, mas, half) for u in us)
    mesh = torch.zeros(N ** 3, dtype=torch.float64, device="cuda")
    for a in range(mas):
        for b in range(mas):
            base = (torch.remainder(fx + a, N) * N + torch.remainder(fy + b, N)) * N
            wab = wx[a] * wy[b]
            for c in range(mas):
                mesh = mesh.index_add(0, base + torch.remainder(fz + c, N), wab * wz[c] * w)
    return mesh.view(N, N, N)


def _window(N, mas, kz):
    w = lambda k: torch.sinc(k.double() / N) ** (-2 * mas)
    return w(_signed(N)), w(kz)


def _combined(fields, N, kz, x0, x1):
    if len(fields) == 1:
        return fields[0][x0:x1]
    ki = _signed(N)
    ph = (ki[x0:x1, None, None] + ki[None, :, None] + kz[None, None, :]).double() * (math.pi / N)
    return 0.5 * (fields[0][x0:x1] + fields[1][x0:x1] * torch.polar(torch.ones_like(ph), ph))


def _pk64(x, y, z, w, N, box, mas, interlace, edges, ells):
    us = [(c * np.float32(N / box)).double() for c in (x, y, z)]     # the estimator's float32 grid coordinates
    w = torch.ones_like(us[0]) if w is None else w.double()
    kz = torch.arange(N // 2 + 1, device="cuda")
    fields, mass = [], None
    for half in ([False, True] if interlace else [False]):
        m = _mesh64(us, w, N, mas, half)
        mass = m.sum() if mass is None else mass
        fields.append(torch.fft.rfftn(m))
        del m
    wx, wz = _window(N, mas, kz)

    def power(x0, x1):
        p = _combined(fields, N, kz, x0, x1).abs() ** 2 * wx[x0:x1, None, None] * wx[None, :, None] * wz[None, None, :]
        if x0 == 0:
            p[0, 0, 0] = 0.0
        return p

    sums, count, ksum = _legendre_sums(power, kz, N, edges)
    pk = sums / count[:, None] * torch.tensor(ELL_FACTORS, device="cuda", dtype=torch.float64) * box ** 3 / mass ** 2
    pk[:, 0] -= box ** 3 * (w * w).sum() / mass ** 2
    for j, ell in enumerate((0, 2, 4)):
        if ell not in ells:
            pk[:, j] *= 0.0                                          # 0, or NaN in an empty bin
    return {"pk": pk, "k_mean": ksum / count * (2.0 * math.pi / box), "nmodes": None}


def _reference_edges(k_edges, box):
    kf = np.float32(np.float32(2.0 * np.pi) / np.float32(box))
    return (np.asarray(k_edges, np.float32) / kf).astype(np.float32), kf


def _powspec64(d, box, k_edges):
    N = d.shape[0]
    e, kf = _reference_edges(k_edges, box)
    kz = torch.arange(N // 2 + 1, device="cuda")
    f = torch.fft.rfftn(d.double())
    wx, wz = _window(N, 2, kz)
    sums, count, _ = _legendre_sums(
        lambda a, b: f[a:b].abs() ** 2 * wx[a:b, None, None] * wx[None, :, None] * wz[None, None, :], kz, N, e)
    pk = sums / count[:, None] * torch.tensor(ELL_FACTORS, device="cuda", dtype=torch.float64) * (box / N ** 2) ** 3
    return torch.from_numpy(0.5 * (e[1:].astype(np.float64) + e[:-1]) * float(kf)).cuda(), pk, count


def _xi64(d, box, s_edges):
    N = d.shape[0]
    f32 = np.float32
    kf = f32(f32(2.0 * np.pi) / f32(box))
    e = (((kf * np.asarray(s_edges, f32)).astype(f32) * f32(N)).astype(f32) / f32(box)).astype(f32)
    e = (e / kf).astype(f32)
    kz = torch.arange(N // 2 + 1, device="cuda")
    wx, wz = _window(N, 2, kz)
    p = torch.fft.rfftn(d.double()).abs() ** 2 * wx[:, None, None] * wx[None, :, None] * wz[None, None, :]
    xi = torch.fft.irfftn(p.to(torch.complex128), s=(N, N, N))
    sums, count, _ = _legendre_sums(lambda a, b: xi[a:b], _signed(N), N, e)
    count = torch.where(count == 0, torch.full_like(count, math.inf), count)
    out = sums / count[:, None] * torch.tensor(ELL_FACTORS, device="cuda", dtype=torch.float64) / float(N) ** 3
    return torch.from_numpy(0.5 * (e[1:].astype(np.float64) + e[:-1]) * (box / N)).cuda(), out, count


def _bispec64(d, box, k1, k2, theta):
    N = d.shape[0]
    f32 = np.float32
    kf = f32(f32(2.0 * np.pi) / f32(box))
    k3 = np.sqrt((f32(k2) * np.sin(theta)) ** 2 + (f32(k2) * np.cos(theta) + f32(k1)) ** 2).astype(f32)
    k_all = np.concatenate([np.array([k1, k2], f32), k3]).astype(f32)
    lo, hi = ((k_all - kf) / kf).astype(f32), ((k_all + kf) / kf).astype(f32)
    kz = torch.arange(N // 2 + 1, device="cuda")
    ki = _signed(N)
    k = (ki[:, None, None] ** 2 + ki[None, :, None] ** 2 + kz[None, None, :] ** 2).float().sqrt()
    a = lambda q: torch.sinc(q.double() / N) ** -2
    dk = torch.fft.rfftn(d.double()) * a(ki)[:, None, None] * a(ki)[None, :, None] * a(kz)[None, None, :]
    fields, norms, P, B = [], [], [], []
    for i in range(len(k_all)):
        m = (k >= float(lo[i])) & (k < float(hi[i]))
        fld = torch.fft.irfftn(torch.where(m, dk, torch.zeros_like(dk)), s=(N, N, N))
        one = torch.fft.irfftn(m.to(torch.complex128), s=(N, N, N))
        P.append((fld ** 2).sum() / (one ** 2).sum() * (box / N ** 2) ** 3)
        if i < 2:
            fields.append(fld)
            norms.append(one)
            if i == 1:
                pair, unit = fields[0] * fields[1], norms[0] * norms[1]
        else:
            B.append((pair * fld).sum() / (unit * one).sum() * (box * box / N ** 3) ** 3)
    P, B = torch.stack(P), torch.stack(B)
    Q = B / (P[0] * P[1] + P[0] * P[2:] + P[1] * P[2:])
    return torch.from_numpy(k_all).cuda().double(), P, torch.from_numpy(theta).cuda().double(), B, Q


def _cic64(x, y, z, N, box):
    """cic_mas_vec of unit weights with wrap, the reference's corner weight (x, y+1, z+1) -> mx my dz included."""
    inv = np.float32(np.float32(1.0) / np.float32(np.float32(box) / np.float32(N)))
    ij, fr = [], []
    for c in (x, y, z):
        u = (c * inv)
        i = u.to(torch.int64)
        d = (u - i.to(torch.float32)).double()
        ij.append(((i, (i + 1) % N)))
        fr.append((1.0 - d, d))
    mesh = torch.zeros(N ** 3, dtype=torch.float64, device="cuda")
    for a in range(2):
        for b in range(2):
            for c in range(2):
                wy = fr[1][0] if (a, b, c) == (0, 1, 1) else fr[1][b]
                ok = (ij[0][a] < N) & (ij[1][b] < N) & (ij[2][c] < N)
                idx = (ij[0][a] * N + ij[1][b]) * N + ij[2][c]
                mesh.index_add_(0, idx[ok], (fr[0][a] * wy * fr[2][c])[ok])
    return mesh.view(N, N, N)


def _grad64(case, st):
    N, box, mas = case["mesh"], case["box"], MAS[case["mas"]]
    kf = np.float32(2.0 * np.pi / box)
    e = np.arange(2.0 * math.pi / box, math.pi * N / box, 2.0 * math.pi / box).astype(np.float32)
    edges = (e / kf).astype(np.float32)
    leaves = [t.detach().double().requires_grad_(True) for t in st["leaves"]]
    w = leaves[3] if len(leaves) > 3 else torch.ones_like(leaves[0])
    us = [t * (N / box) for t in leaves[:3]]
    kz = torch.arange(N // 2 + 1, device="cuda")
    fields, mass = [], None
    for half in ([False, True] if case["interlace"] else [False]):
        m = _mesh64(us, w, N, mas, half)
        mass = m.sum() if mass is None else mass
        fields.append(torch.fft.rfftn(m))
    wx, wz = _window(N, mas, kz)
    p = _combined(fields, N, kz, 0, N).abs().square() * wx[:, None, None] * wx[None, :, None] * wz[None, None, :]
    ki = _signed(N)
    k2 = ki[:, None, None] ** 2 + ki[None, :, None] ** 2 + kz[None, None, :] ** 2
    mu2 = ((kz[None, None, :] ** 2).double() / k2.clamp(min=1).double()).reshape(-1)
    b = _bin_of_k2(edges, 3 * (N // 2) ** 2)[k2.reshape(-1)]
    keep = (b >= 0) & (k2.reshape(-1) > 0)
    bb, pf, mu2 = b[keep], p.reshape(-1)[keep], mu2[keep]
    count = torch.bincount(bb, minlength=len(edges) - 1).double()
    pk = []
    for f, lg in zip(ELL_FACTORS, (torch.ones_like(mu2), 1.5 * mu2 - 0.5, (35 * mu2 * mu2 - 30 * mu2 + 3) / 8)):
        s = torch.zeros(len(edges) - 1, dtype=torch.float64, device="cuda").index_add(0, bb, pf * lg)
        pk.append(f * s / count * box ** 3 / mass ** 2)
    pk[0] = pk[0] - box ** 3 * (w * w).sum() / mass ** 2
    pk = torch.stack(pk, dim=1)
    return {"pk": pk.detach(), "grads": _fit_grads(pk, st["target"], leaves)}


def exact(case, seed):
    kind = case["kind"]
    gen = _generator(seed)
    if kind == "pk":
        x, y, z, w = _catalogue(case["n"], case["box"], gen, case["weights"])
        return _pk64(x, y, z, w, case["mesh"], case["box"], MAS[case["mas"]], case["interlace"], _edges_kf(case),
                     _ells(case))
    if kind == "batch":
        edges = np.arange(1, case["mesh"] // 2).astype(np.float32)
        got = [_pk64(*_catalogue(n, case["box"], gen), case["mesh"], case["box"], MAS[case["mas"]], case["interlace"],
                     edges, _ells(case)) for n in _counts(case)]
        return {"pk": torch.stack([r["pk"] for r in got]), "k_mean": torch.stack([r["k_mean"] for r in got]),
                "nmodes": None}
    if kind == "deposit":
        x, y, z, _ = _catalogue(case["n"], case["box"], gen)
        return _cic64(x, y, z, case["mesh"], case["box"])
    if kind in ("powspec", "xi", "bispec"):
        d = _contrast(case["mesh"], case["box"], gen)
        if kind == "powspec":
            return _powspec64(d, case["box"], _k_edges(case))
        if kind == "xi":
            return _xi64(d, case["box"], _s_edges(case))
        return _bispec64(d, case["box"], case["k1"], case["k2"], _theta(case))
    return _grad64(case, prepare(case, seed))
