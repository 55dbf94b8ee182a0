"""Spilled bucket entries: the tiles collect them from lists (many modest clumps) or by looking through all
spilled entries (one tile that holds most of them); either way the same bits as buckets that hold everything."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N, BOX = 64, 300.0


def _catalogue(n_bg, clumps, per, seed):
    rng = np.random.default_rng(seed)
    H = BOX / N
    at = rng.integers(0, N, (3, clumps)) * H
    p = np.concatenate([rng.random((3, n_bg)) * BOX,
                        np.repeat(at, per, axis=1) + rng.random((3, clumps * per)) * 0.9 * H], axis=1)
    return [torch.from_numpy(a.astype(np.float32)).cuda() for a in p[:, rng.permutation(p.shape[1])]]


@pytest.mark.parametrize("clumps,per", [(1, 2500), (1, 40_000), (200, 700), (3, 5000), (40, 3000)])
@pytest.mark.parametrize("interlace", [False, True])
def test_spilled_entries_change_no_bit(clumps, per, interlace):
    from gbpowspec import PkConfig, PowerSpectrum, _lib, read_stats
    from gbpowspec.batch import BatchRunner, ParticleArena
    x, y, z = _catalogue(20_000, clumps, per, seed=clumps + per)
    cfg = PkConfig(n_mesh=N, box_size=BOX, mas="tsc", interlace=interlace)
    r = PowerSpectrum(cfg).run(x, y, z)
    torch.cuda.synchronize()
    assert read_stats(r.stats).flags & _lib.STATS_REFILLED
    arena = ParticleArena([tuple(t.cpu().numpy() for t in (x, y, z))])
    arena.upload()
    big = BatchRunner(N, capacity=200 * x.numel(), mas="tsc", interlace=interlace, ells=(0, 2, 4),
                      kedges_grid=cfg.kedges_grid(), n_lanes=1, tiles=None)
    res = big.run(arena.job_table(BOX, N))
    torch.cuda.synchronize()
    assert res.deposit_stats()[0].flags & _lib.STATS_REFILLED == 0
    assert torch.equal(res.pk[0], r.pk) and torch.equal(res.nmodes[0], r.nmodes)
    assert res.deposit_stats()[0].mass[0] == read_stats(r.stats).mass[0]
    big.close()
