"""Workspace of the mesh deposit: room for the buckets and for the surplus of the most clustered catalogue, no more
than one 16-byte entry per particle and tile it can touch takes, plus the counters (host arithmetic, no GPU)."""
import pytest


@pytest.mark.parametrize("n,N,mas,interlace,compat", [(4 << 20, 512, 2, False, 1), (16 << 20, 512, 2, False, 1),
                                                      (1_500_007, 360, 2, True, 0), (1 << 27, 1024, 4, True, 0),
                                                      (1 << 20, 128, 3, False, 0)])
def test_deposit_workspace_is_an_entry_per_tile_a_particle_can_touch(n, N, mas, interlace, compat):
    from gbpowspec import _native
    tiles = (-(-N // 16)) ** 3
    assert _native.deposit_workspace_size(n, N, mas, interlace, compat) <= 8 * 16 * n + 512 * tiles
