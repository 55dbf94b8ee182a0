"""The packed transform's kernels at 512^3 and 1024^3, which are other code than at smaller sides (two warps per
column, named barriers, one plane per block): the bispectrum against the cuFFT path, xi's shells against the field
and float64, the adjoint against the standard one, P_l of two grids against the standard transform, each by the
test of the smaller sides and with its bounds."""
import numpy as np
import pytest
import torch

import test_gpu_bispec_limits
import test_gpu_grad_packed
import test_gpu_planes
import test_gpu_xi_shells

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _memory():
    torch.cuda.empty_cache()
    yield
    torch.cuda.empty_cache()


@pytest.mark.parametrize("N,k1,k2,angles", [(512, 12.0, 17.0, 7), (512, 190.0, 230.0, 3), (1024, 30.0, 41.0, 4)])
def test_bispectrum(monkeypatch, N, k1, k2, angles):
    test_gpu_bispec_limits.test_outermost_shell_reaches_the_last_edge(monkeypatch, N, k1, k2, angles)


@pytest.mark.parametrize("N,edges", [(512, np.arange(0.0, 60.0, 2.5)), (512, "cube"), (1024, np.arange(0.0, 40.0, 4.0)),
                                     (1024, "half")])
def test_xi(N, edges):
    test_gpu_xi_shells.test_shells_match_the_field(N, edges, 1)


@pytest.mark.parametrize("N,G,edges", [(512, 1, "nyquist"), (512, 2, "nyquist"), (512, 1, "corner"), (512, 2, "corner"),
                                       (1024, 1, "corner"), (1024, 2, "low"), (1024, 2, "nyquist")])
def test_adjoint(N, G, edges):
    test_gpu_grad_packed.test_packed_adjoint_matches_the_standard_one(N, G, edges)


@pytest.mark.parametrize("N", [512, 1024])
@pytest.mark.parametrize("last", ["block", "corner"])
def test_two_grids(N, last):
    test_gpu_planes.test_interleaved_planes(N, 2, last)
