"""gbp_xi_shells against gbp_xi and a float64 evaluation of the same mesh: equal cell counts, equal NaNs, and
shell sums no further from float64 than 1.5 times gbp_xi's (the worst bin of each multipole, relative to the
largest value of the field, which sets the round-off of both), for a few short shells, shells past half the
box, all of the cube and none, with and without the NaN at r = 0."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 128, 256])
@pytest.mark.parametrize("edges", [np.arange(0.0, 6.5, 1.5), np.arange(1.0, 30.0, 1.0), "half", "cube", [0.2, 0.7]])
@pytest.mark.parametrize("nan_origin", [0, 1])
def test_shells_match_the_field(N, edges, nan_origin):
    from gbpowspec import _lib, _native
    dev = torch.device("cuda", 0)
    if isinstance(edges, str):
        edges = np.arange(0.0, {"half": 0.55, "cube": 0.9}[edges] * N, 2.0)
    gen = torch.Generator(device="cuda").manual_seed(N)
    d = torch.randn((N, N, N), generator=gen, device=dev)
    plan, bins = _native.fft_plan(N, 1, dev), _native.bins_for(np.asarray(edges, np.float32), N, dev)
    lib, st, need, p = _lib.load(), _native._stream_of(dev), C.c_size_t(0), lambda t: C.c_void_p(t.data_ptr())
    spec, field = torch.empty(plan.spectrum_floats, device=dev), torch.empty_like(d)
    out = []
    for fused in (False, True):
        sums = torch.full((bins.n_bins, 3), 7.0, dtype=torch.float64, device=dev)
        counts = torch.full((bins.n_bins,), 7, dtype=torch.int64, device=dev)
        size = lib.gbp_xi_shells_workspace_size if fused else lib.gbp_xi_workspace_size
        _lib.check(size(plan.handle, bins.handle, C.byref(need)), "size")
        ws = _native.workspace(need.value, dev).fill_(255)
        if fused:
            r = lib.gbp_xi_shells(plan.handle, p(d), p(spec), bins.handle, 2, nan_origin, p(sums), p(counts), p(ws),
                                  ws.numel(), st)
        else:
            r = lib.gbp_xi(plan.handle, p(d), p(spec), p(field), bins.handle, 2, nan_origin, p(sums), p(counts),
                           p(ws), ws.numel(), st)
        _lib.check(r, "xi")
        torch.cuda.synchronize()
        out.append((sums.cpu().numpy(), counts.cpu().numpy()))
    (a, ca), (b, cb) = out
    np.testing.assert_array_equal(ca, cb)
    np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
    want, peak = _float64(d, np.asarray(edges, np.float32))
    for l in range(3):
        ea, eb = (np.nanmax(np.abs(v[:, l] - want[:, l]), initial=0.0) / peak for v in (a, b))
        assert eb <= 1.5 * ea + 1e-7, (l, ea, eb)          # 1e-7: a float32 ulp of the peak


def _float64(d, edges):
    """[nb, 3] sums of N^3 xi L_l over the shells in float64, and the field's largest value."""
    N = d.shape[0]
    i = torch.arange(N, device=d.device)
    s = torch.where(i > N // 2, i - N, i)
    win = lambda k: torch.sinc(k.double() / N) ** -4
    p = torch.fft.rfftn(d.double()).abs() ** 2
    p = p * win(s)[:, None, None] * win(s)[None, :, None] * win(i[: N // 2 + 1])[None, None, :]
    f = torch.fft.irfftn(p.to(torch.complex128), s=(N, N, N)) * N ** 3
    r2 = s[:, None, None] ** 2 + s[None, :, None] ** 2 + s[None, None, :] ** 2
    mu2 = ((s ** 2)[None, None, :].double() / r2.clamp(min=1).double()).reshape(-1)
    e = torch.from_numpy(edges).to(d.device)
    r = r2.to(torch.float32).sqrt().reshape(-1)
    b = torch.searchsorted(e, r, right=True) - 1
    b = torch.where(r == e[-1], torch.full_like(b, e.numel() - 2), b)
    keep = (b >= 0) & (b < e.numel() - 1)
    b, v, m = b[keep], f.reshape(-1)[keep], mu2[keep]
    legendre = (torch.ones_like(m), 1.5 * m - 0.5, (35 * m * m - 30 * m + 3) / 8)
    sums = [torch.zeros(e.numel() - 1, dtype=torch.float64, device=d.device).index_add_(0, b, v * q) for q in legendre]
    return torch.stack(sums, 1).cpu().numpy(), float(f.abs().max())
