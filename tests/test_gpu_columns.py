"""The column buckets (each particle written once, nine runs per tile) against the mesh deposit on the same
particles: the exact totals and the kept counts, P_l to float32 round-off, for every tile shape, scheme and
grid count, with particles on cell and tile faces, at the box's edge and outside it, one particle, and n = 0."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("mas", ["ngp", "cic", "tsc", "pcs"])
@pytest.mark.parametrize("interlace", [False, True])
@pytest.mark.parametrize("n", [0, 1, 777, 60_000])
def test_column_buckets_match_the_mesh_deposit(N, mas, interlace, n):
    from gbpowspec import PkConfig, PowerSpectrum, _lib, _native, read_stats
    box = float(N)                                            # cells of 1: faces are exact floats
    rng = np.random.default_rng(N + n)
    p = rng.random((3, n)) * 3 * box - box
    p[:, ::3] = np.round(p[:, ::3] * 2) / 2                   # on nodes and half-way between them
    x, y, z = (torch.from_numpy(a.astype(np.float32)).cuda() for a in p)
    cfg = PkConfig(n_mesh=N, box_size=box, mas=mas, interlace=interlace)
    mesh, st = _native.deposit(x, y, z, None, n_mesh=N, inv_cell=1.0, mas=cfg.mas_order, interlace=interlace)
    plan, bins = _native.fft_plan(N, cfg.grids, x.device), _native.bins_for(cfg.kedges_grid(), N, x.device)
    want = _native.fft_power(plan, mesh, torch.empty(plan.spectrum_floats, device="cuda"), bins,
                             mas_order=cfg.mas_order, ells=cfg.ells_mask(), mass=st)
    torch.cuda.synchronize()
    a, w = read_stats(st), want.sums.cpu().numpy()
    for tiles in _native.tile_variants(N):
        ps = PowerSpectrum(cfg, tiles=tiles)
        r = ps.run(x, y, z)
        torch.cuda.synchronize()
        b = read_stats(r.stats)
        assert b.n_kept == a.n_kept == n and b.sum_w == a.sum_w and b.sum_w2 == a.sum_w2
        # a contribution is quantised at 2^-18 or finer in the fused tiles, 2^-30 in the mesh
        np.testing.assert_allclose(b.mass[:], a.mass[:], rtol=1e-6)
        got = ps.sums.sums.cpu().numpy()
        assert np.all(np.abs(got - w) <= 2e-6 * np.abs(w[:, :1]) + 1e-300), tiles
