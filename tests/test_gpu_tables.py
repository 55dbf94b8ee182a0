"""Host tables of the drop-ins: each queued call keeps its own."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 48])
def test_tables_of_queued_calls(n):
    """Calls queued behind a long one return the bin centres of their own box, not of a later call's."""
    from gbpowspec import powspec_vec
    gen = torch.Generator(device="cuda").manual_seed(3)
    delta = torch.randn((n, n, n), generator=gen, device="cuda")
    a = torch.randn((8192, 8192), device="cuda")
    boxes = [300.0 + 7.0 * i for i in range(24)]
    edges = [(np.arange(1, n // 2) * np.float32(2 * np.pi / b)).astype(np.float32) for b in boxes]
    alone = []
    for b, e in zip(boxes, edges):
        alone.append([t.cpu() for t in powspec_vec(delta, b, e)])
    torch.cuda.synchronize()
    for _ in range(20):
        a = a @ a * 1e-4                    # the calls below are enqueued while this runs
    queued = [powspec_vec(delta, b, e) for b, e in zip(boxes, edges)]
    for want, got in zip(alone, queued):
        for w, g in zip(want, got):
            assert torch.equal(torch.nan_to_num(w), torch.nan_to_num(g.cpu()))
