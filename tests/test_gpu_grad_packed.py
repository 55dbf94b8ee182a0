"""The adjoint on the packed spectrum (gbp_power_backward_packed) against the adjoint on the standard one
(gbp_power_backward: half spectra, cuFFT inverse): the gradient meshes agree to float32 round-off of the
transforms, 2e-6 of their norm, for edges up to k_Nyquist, for a few low bins and for edges that take in
the Nyquist planes and the corners of the cube."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [64, 128, 256])
@pytest.mark.parametrize("G", [1, 2])
@pytest.mark.parametrize("edges", ["nyquist", "low", "corner"])
def test_packed_adjoint_matches_the_standard_one(N, G, edges):
    from gbpowspec import _lib, _native
    dev = torch.device("cuda", 0)
    e = {"nyquist": np.arange(1, N // 2), "low": np.arange(1, 9, 2),
         "corner": np.arange(1, int(0.9 * N))}[edges].astype(np.float32)
    gen = torch.Generator(device="cuda").manual_seed(N + G)
    mesh = torch.rand((G, N, N, N), generator=gen, device=dev) + 0.5
    plan, bins = _native.fft_plan(N, G, dev), _native.bins_for(e, N, dev)
    mask = _lib.ELL0 | _lib.ELL2 | _lib.ELL4
    mass = torch.stack([mesh[0].double().sum(), mesh[-1].double().sum()])
    p = lambda t: C.c_void_p(t.data_ptr())
    lib, st = _lib.load(), _native._stream_of(dev)
    packed = torch.empty(plan.spectrum_floats, device=dev)
    sums = _native.fft_power(plan, mesh, packed, bins, mas_order=3, ells=mask, mass=mass)
    pk, _ = _native.normalize(sums, n_mesh=N, box_size=500.0, mass=mass)
    spec = torch.empty_like(packed)
    plan.execute(mesh, spec)
    g = torch.randn((bins.n_bins, 3), generator=gen, device=dev, dtype=torch.float64)
    need = C.c_size_t(0)
    want, got = torch.empty_like(mesh), torch.full_like(mesh, float("nan"))
    _lib.check(lib.gbp_power_backward_workspace_size(plan.handle, C.byref(need)), "size")
    ws = _native.workspace(need.value, dev)
    _lib.check(lib.gbp_power_backward(p(spec), plan.handle, bins.handle, 3, p(g), p(sums.nmodes), p(mass), 500.0,
                                      p(want), p(ws), ws.numel(), st), "standard")
    _lib.check(lib.gbp_power_backward_packed_workspace_size(plan.handle, bins.handle, C.byref(need)), "size")
    ws = _native.workspace(need.value, dev).fill_(255)                     # NaN wherever nothing is written
    scal = torch.empty(2, dtype=torch.float64, device=dev)
    keep = packed.clone()
    _lib.check(lib.gbp_power_backward_packed(p(packed), plan.handle, bins.handle, 3, p(g), p(pk), p(sums.nmodes),
                                             p(mass), 500.0, 1, p(got), p(scal), p(ws), ws.numel(), st), "packed")
    torch.cuda.synchronize()
    assert torch.equal(packed.view(torch.int32), keep.view(torch.int32))   # read only
    for a, b in zip(got.double(), want.double()):
        assert float((a - b).norm() / b.norm()) < 2e-6
    full = sums.nmodes > 0
    m, box3 = float(mass[0]), 500.0 ** 3
    np.testing.assert_allclose(float(scal[0]), float((g * (-2.0 * pk / m))[full].sum()), rtol=1e-12)
    np.testing.assert_allclose(float(scal[1]), -2.0 * box3 / m ** 2 * float(g[full, 0].sum()), rtol=1e-12)
