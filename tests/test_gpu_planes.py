"""Packed spectra with interleaved x planes: gbp_fft_power against gbp_fft_r2c + gbp_power where rows, planes and
kz blocks end: edges that stop inside a block of kz, that take in the Nyquist planes, and the largest mesh with one
grid.  The same modes, and sums equal to the float32 round-off of the two transforms (the bound of the fused path)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,G", [(64, 1), (64, 2), (128, 1), (256, 2), (512, 1), (1024, 1)])
@pytest.mark.parametrize("last", ["block", "corner"])
def test_interleaved_planes(N, G, last):
    from gbpowspec import _lib, _native
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device="cuda").manual_seed(N + G)
    mesh = torch.rand((G, N, N, N), generator=gen, device=dev) + 0.5
    edges = np.linspace(1.0, 12.5 if last == "block" else 0.86 * N, 14).astype(np.float32)
    plan, bins = _native.fft_plan(N, G, dev), _native.bins_for(edges, N, dev)
    spec = torch.empty(plan.spectrum_floats, device=dev)
    mask = _lib.ELL0 | _lib.ELL2 | _lib.ELL4
    plan.execute(mesh, spec)
    want = _native.power(spec, G, bins, mas_order=2, ells=mask, z_pitch=plan.pitch)
    spec.fill_(float("nan"))                       # nothing is read that was not written
    got = _native.fft_power(plan, mesh, spec, bins, mas_order=2, ells=mask)
    torch.cuda.synchronize()
    assert torch.equal(got.nmodes, want.nmodes)
    w, g = want.sums.cpu().numpy(), got.sums.cpu().numpy()
    assert np.all(np.abs(g - w) <= 2e-6 * np.abs(w[:, :1]))
