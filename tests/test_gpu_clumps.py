"""Catalogues whose particles lie in a few dense clumps: the surplus of their buckets is found again in a time that
does not depend on how many clumps there are, and changes no bit.

* time: eight clumps cost about what one does, and less than in proportion to the largest clump (a serial walk of
  a tile's surplus by a few threads cost four times as much as the deposit itself);
* bits: the mesh and the totals of a clumped catalogue against the same particles in a workspace whose buckets hold
  everything, for the schemes whose weights are rounded products, jobs and weights included."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _clumps(N, n_bg, clumps, per, seed, box):
    rng = np.random.default_rng(seed)
    at = rng.integers(0, N, (3, clumps))
    p = np.concatenate([rng.random((3, n_bg)) * N, np.repeat(at, per, axis=1) + rng.random((3, clumps * per)) * 0.9],
                       axis=1)[:, rng.permutation(n_bg + clumps * per)] % N
    return [torch.from_numpy((a * box / N).astype(np.float32)).cuda() for a in p]


def _ms(f, reps=5):
    f()
    torch.cuda.synchronize()
    ts = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        b.synchronize()
        ts.append(a.elapsed_time(b))
    return float(np.median(ts))


def test_surplus_is_collected_in_parallel():
    """16 clumps of 65,536 against one of 65,536: sixteen tiles side by side, not one after the other; the walk of
    lists took 5 times as long for the 16, a sixteenth of all surplus each."""
    from gbpowspec import cic_mas_vec
    N = 256
    mesh = torch.zeros((N, N, N), device="cuda")

    def ms(clumps):
        x, y, z = _clumps(N, 200_000, clumps, 65_536, 3, float(N))
        w = torch.ones_like(x)
        return _ms(lambda: cic_mas_vec(mesh, x, y, z, w, x.numel(), 0.0, 0.0, 0.0, float(N), N, True))
    one, many = ms(1), ms(16)
    assert many < 2.0 * one + 0.2, (one, many)


def test_dense_tiles_of_small_meshes_are_visited_once():
    """Eight clumps of 98,304 particles at 128^3, one grid: two visits of each dense tile's entries took 10.1 ms,
    one takes 6.0."""
    from gbpowspec import PkConfig, PowerSpectrum
    N, n = 128, 98_304
    x, y, z = _clumps(N, 262_144, 8, n, 7, float(N))
    ps = PowerSpectrum(PkConfig(n_mesh=N, box_size=float(N), mas="cic", interlace=False))
    assert _ms(lambda: ps.run(x, y, z)) < 8.0


@pytest.mark.parametrize("mas,interlace", [("ngp", False), ("cic", True), ("tsc", False), ("pcs", False),
                                           ("pcs", True)])
@pytest.mark.parametrize("N,clumps,per", [(48, 5, 6000), (64, 1, 30_000), (64, 30, 900), (128, 40, 3000)])
def test_spilled_particles_change_no_bit(N, clumps, per, mas, interlace):
    from gbpowspec import PkConfig, PowerSpectrum, _lib, _native, read_stats
    from gbpowspec.batch import BatchRunner, ParticleArena
    box = 300.0
    x, y, z = _clumps(N, 15_000, clumps, per, N + clumps, box)
    n = x.numel()
    w = torch.rand(n, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda") - 0.25
    arena = ParticleArena([tuple(t.cpu().numpy() for t in (x, y, z, w))])
    arena.upload()
    jobs = arena.job_table(box, N)
    order = {"ngp": 1, "cic": 2, "tsc": 3, "pcs": 4}[mas]
    inv = float(np.float32(N / box))
    mesh, st = _native.deposit(x, y, z, w, n_mesh=N, inv_cell=inv, mas=order, interlace=interlace)
    lib, cap, need = _lib.load(), 200 * n, C.c_size_t(0)
    _lib.check(lib.gbp_deposit_workspace_size(cap, N, order, int(interlace), 0, C.byref(need)), "size")
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    out, st2 = torch.empty_like(mesh), torch.empty_like(st)
    p = lambda t: C.c_void_p(t.data_ptr())
    _lib.check(lib.gbp_deposit_job(p(jobs), cap, N, order, int(interlace), p(out), p(st2), p(ws), ws.numel(),
                                   C.c_void_p(torch.cuda.current_stream().cuda_stream)), "gbp_deposit_job")
    torch.cuda.synchronize()
    a, b = read_stats(st), read_stats(st2)
    assert torch.equal(mesh, out) and list(a.mass) == list(b.mass) and a.n_kept == b.n_kept == n
    assert b.flags & _lib.STATS_REFILLED == 0
    del ws
    if not _native.tile_variants(N):
        return
    cfg = PkConfig(n_mesh=N, box_size=box, mas=mas, interlace=interlace)
    for tiles in _native.tile_variants(N):
        r = PowerSpectrum(cfg, tiles=tiles).run(x, y, z, w)
        small = BatchRunner(N, capacity=n, mas=mas, interlace=interlace, ells=(0, 2, 4),
                            kedges_grid=cfg.kedges_grid(), n_lanes=1, tiles=tiles)
        big = BatchRunner(N, capacity=cap, mas=mas, interlace=interlace, ells=(0, 2, 4),
                          kedges_grid=cfg.kedges_grid(), n_lanes=1, tiles=tiles)
        rs, rb = small.run(jobs), big.run(jobs)
        torch.cuda.synchronize()
        for q in (rs, rb):
            assert torch.equal(q.pk[0], r.pk), tiles
            assert list(q.deposit_stats()[0].mass) == list(read_stats(r.stats).mass), tiles
        small.close()
        big.close()


def test_fused_workspace_and_limits():
    """What the fused path takes: the buckets (twice the catalogue), a table for the surplus and little else, for
    every tile shape; a catalogue is refused only when an entry per tile it can touch has no 32-bit number (one grid
    of NGP touches one tile, other schemes four)."""
    from gbpowspec import _lib, _native
    dev = torch.device("cuda", 0)
    lib = _lib.load()
    size = C.c_size_t(0)

    def need(N, n, mas, grids, tiles=None):
        plan = _native.FFTPlan(N, grids, dev)
        if tiles:
            plan.set_tiles(*tiles)
        bins = _native.bins_for(np.arange(1, N // 2).astype(np.float32), N, dev)
        st = lib.gbp_particles_power_workspace_size(n, plan.handle, bins.handle, mas, 7, C.byref(size))
        plan.close()
        return st, size.value
    for N, n, mas, grids in ((512, 4 << 20, 3, 2), (256, 1 << 20, 3, 2), (128, 1 << 20, 2, 2), (128, 1 << 20, 2, 1),
                             (1024, 16 << 20, 4, 2)):
        for tiles in _native.tile_variants(N):
            st, b = need(N, n, mas, grids, tiles)
            assert st == 0 and b <= 72 * n + 4096 * (N // 4) ** 2, (N, tiles, b / n)
    assert need(512, 4_200_000_000, 1, 1)[0] == 0
    assert need(512, 2_000_000_000, 1, 1)[0] == 0
    assert need(512, 1_070_000_000, 2, 1)[0] == 0
    for mas, grids, n in ((1, 1, 4_294_967_295), (1, 2, 1_080_000_000), (2, 1, 1_080_000_000)):
        assert need(512, n, mas, grids)[0] == _lib.GBP_ERR_UNSUPPORTED
