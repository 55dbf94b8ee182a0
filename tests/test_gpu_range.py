"""Power spectra whose modes square to float32 values near the largest: finite on the packed transform wherever
they are on the standard one, and equal to the float32 round-off of the transforms.  A mode that carried a factor 2
(one grid) or 4 (two) until it was squared overflowed at |F| > 9.2e18 or 4.6e18; the standard path squares F itself
(1.8e19), or the sum of two grids' modes (9.2e18)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 128])
@pytest.mark.parametrize("G", [1, 2])
@pytest.mark.parametrize("largest", [0.8, 5e-20, 1e-37])
def test_large_and_small_modes(N, G, largest):
    from gbpowspec import _lib, _native
    dev = torch.device("cuda", 0)
    amplitude = largest * {1: 1.8e19, 2: 9.2e18}[G]
    i = torch.arange(N, device=dev, dtype=torch.float64) * (2 * np.pi / N)
    wave = torch.cos(3 * i[:, None, None] + 2 * i[None, :, None] + 5 * i[None, None, :])
    one = (wave * (2.0 * amplitude / N ** 3)).float()                     # |F| = amplitude at (3, 2, 5) and its mirror
    mesh = one.repeat(G, 1, 1, 1).contiguous()
    if G == 2:                                                            # the second grid, half a cell on
        mesh[1] = (torch.cos(3 * i[:, None, None] + 2 * i[None, :, None] + 5 * i[None, None, :] - 10 * np.pi / N)
                   * (2.0 * amplitude / N ** 3)).float()
    plan, bins = _native.fft_plan(N, G, dev), _native.bins_for(np.array([5.5, 7.0], np.float32), N, dev)
    spec = torch.empty(plan.spectrum_floats, device=dev)
    mask = _lib.ELL0 | _lib.ELL2 | _lib.ELL4
    plan.execute(mesh, spec)
    want = _native.power(spec, G, bins, mas_order=0, ells=mask, z_pitch=plan.pitch)
    got = _native.fft_power(plan, mesh, spec, bins, mas_order=0, ells=mask)
    torch.cuda.synchronize()
    w, g = want.sums.cpu().numpy(), got.sums.cpu().numpy()
    assert np.all(np.isfinite(w)) and w[0, 0] > 0.5 * amplitude ** 2
    assert np.all(np.abs(g - w) <= 4e-6 * w[0, 0])
