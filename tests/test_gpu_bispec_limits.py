"""gbp_bispec with the sorted shell limits alone as edges, as its header states the contract: the last elementary
bin belongs to the outermost shell (the wrapper appends an edge and never gets there).  The packed path against the
cuFFT path: equal mode counts, P of every shell to 5e-6 of its own value (sums of squares: the round-off of two
float32 transforms), B to 5e-6 of the largest."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,k1,k2,angles", [(64, 3.0, 4.0, 5), (64, 28.0, 24.0, 6), (128, 20.0, 33.0, 9)])
def test_outermost_shell_reaches_the_last_edge(monkeypatch, N, k1, k2, angles):
    from gbpowspec import _lib, _native, correlations
    dev = torch.device("cuda", 0)
    box = 2 * np.pi * 100.0                                                # kF = 0.01
    gen = torch.Generator(device="cuda").manual_seed(N + angles)
    d = torch.exp(0.5 * torch.randn((N, N, N), generator=gen, device=dev))
    d = (d / d.mean() - 1.0).contiguous()
    theta = np.linspace(0.1, 3.0, angles).astype(np.float32)
    _, lo, hi, _ = correlations.bispec_shells(box, 0.01 * k1, 0.01 * k2, theta)
    edges, shells = correlations._elementary_bins(lo, hi)
    edges = edges[:-1]
    S = len(shells)
    assert shells.max() == len(edges) - 1                                  # one past the last bin
    sb = torch.from_numpy(shells).to(dev)
    bins = _native.Bins(edges, N, dev)
    monkeypatch.setenv("GBP_FFT_BACKEND", "cufft")
    cufft = _native.FFTPlan(N, 1, dev)
    monkeypatch.delenv("GBP_FFT_BACKEND")
    lib, p = _lib.load(), lambda t: C.c_void_p(t.data_ptr())
    out = []
    for plan in (cufft, _native.fft_plan(N, 1, dev)):
        need = C.c_size_t(0)
        _lib.check(lib.gbp_bispec_workspace_size(plan.handle, bins.handle, C.byref(need)), "size")
        ws = _native.workspace(need.value, dev)
        spec = torch.empty(plan.spectrum_floats, device=dev)
        pk, bk, qk = (torch.empty(S, dtype=torch.float64, device=dev) for _ in range(3))
        nm = torch.empty(S, dtype=torch.int64, device=dev)
        _lib.check(lib.gbp_bispec(plan.handle, p(d), p(spec), bins.handle, 2, p(sb), S, box, p(pk), p(bk), p(qk),
                                  p(nm), p(ws), ws.numel(), _native._stream_of(dev)), "gbp_bispec")
        torch.cuda.synchronize()
        out.append((nm.cpu().numpy(), pk.cpu().numpy(), bk[: S - 2].cpu().numpy()))
    (n0, p0, b0), (n1, p1, b1) = out
    np.testing.assert_array_equal(n1, n0)
    np.testing.assert_allclose(p1, p0, rtol=5e-6)
    assert np.max(np.abs(b1 - b0)) <= 5e-6 * np.max(np.abs(b0))
    bins.close()
    cufft.close()
