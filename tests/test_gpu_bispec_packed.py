"""The bispectrum on the packed transform against the cuFFT path (plans forced to cuFFT) and the float64
oracle: equal mode counts, P and B no further from float64 than 1.5 times the cuFFT path's worst shell plus
1e-6, for shells near k = 0, overlapping ones, odd window orders, and shells in the corners of the cube."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,k1,k2,angles,mas", [(64, 3.0, 4.0, 5, 2), (64, 12.0, 12.0, 7, 3), (64, 28.0, 24.0, 6, 1),
                                                (128, 20.0, 33.0, 9, 2), (128, 60.0, 50.0, 4, 4)])
def test_packed_matches_cufft_and_float64(monkeypatch, N, k1, k2, angles, mas):
    from gbpowspec import _native, bispectrum
    from oracle import truth_f64 as T
    box = 2 * np.pi * 100.0                                                # kF = 0.01
    gen = torch.Generator(device="cuda").manual_seed(N + angles)
    g = torch.randn((N, N, N), generator=gen, device="cuda")
    d = torch.exp(0.5 * g)
    d = (d / d.mean() - 1.0).contiguous()
    theta = np.linspace(0.1, 3.0, angles).astype(np.float32)
    args = (box, 0.01 * k1, 0.01 * k2, theta)
    got = bispectrum(d, *args, mas_order=mas)
    dev = d.device
    monkeypatch.setenv("GBP_FFT_BACKEND", "cufft")
    cufft = _native.FFTPlan(N, 1, dev)
    monkeypatch.delenv("GBP_FFT_BACKEND")
    monkeypatch.setattr(_native, "fft_plan", lambda *a: cufft)
    old = bispectrum(d, *args, mas_order=mas)
    torch.cuda.synchronize()
    _, p, b, _, nm = T.bispec(d.cpu().numpy(), *args, mas_order=mas)
    assert torch.equal(got[4], old[4])
    np.testing.assert_array_equal(got[4].cpu().numpy(), nm)
    for i, want in ((1, p), (2, b)):
        e_new, e_old = (np.max(np.abs(v[i].cpu().numpy() - want)) / np.max(np.abs(want)) for v in (got, old))
        assert e_new <= 1.5 * e_old + 1e-6, (i, e_new, e_old)
    cufft.close()
