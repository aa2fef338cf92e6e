"""Outputs of the modular products whose elements the operands' integers
cannot hold: recomputed in FP64, never taken for exact zeros."""
import numpy as np
import pytest
import torch

from test_gpu_mod import _bound, _gemm

pytestmark = pytest.mark.gpu


def _both(lib, A, B):
    """The modular product and the FP64 kernel's, both within a
    componentwise bound of sums in any order."""
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    C = torch.zeros(A.shape[0], B.shape[1], dtype=torch.float64, device="cuda")
    got, ref = _gemm(lib, 1, Ad, Bd, C), _gemm(lib, 0, Ad, Bd, C)
    tol = 2 * _bound(Ad, Bd) + 2e-323
    worst = ((got - ref).abs() / tol).max()
    assert bool(((got - ref).abs() <= tol).all()), float(worst)


@pytest.mark.parametrize("K", [200, 700])
@pytest.mark.parametrize("far", [1e-12, 1e-16, 1e-17, 1e-18, 1e-19, 1e-25, 1e-150, 1e-310])
def test_elements_below_the_integers(gpulib, far, K):
    """The large elements of A meet the small ones of B, which vanish from
    the integers (below ~2^-62 of their row's norm, 2e-19) at some of these."""
    rng = np.random.default_rng(K)
    A, B = rng.standard_normal((70, K)), rng.standard_normal((K, 90))
    A[:, ::2] *= far
    B[1::2] *= far
    _both(gpulib, A, B)


@pytest.mark.parametrize("place", [40, 56, 59, 61])
def test_small_products_that_cancel(gpulib, place):
    """Two small elements per row (and the large ones meeting zeros): their
    products' squares underflow FP32 and their integers' sum can cancel."""
    rng = np.random.default_rng(place)
    A, B = np.zeros((300, 40)), np.zeros((40, 300))
    A[:, 0], B[1] = 1.0, 1.0
    A[:, 2:4] = 2.0 ** -place * (1.0 + rng.random((300, 2)))
    B[2:4] = 2.0 ** -place * (1.0 + rng.random((2, 300))) * np.array([[1.0], [-1.0]])
    _both(gpulib, A, B)


def test_true_zeros_stay_zeros(gpulib):
    """Disjoint supports, empty rows and columns: zeros, with elements below
    the integers beside them or not."""
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal((100, 64)), rng.standard_normal((64, 70))
    A[:, 32:] = 0.0
    B[:32] = 0.0
    A[7], B[:, 5] = 0.0, 0.0
    A[:50, :8] *= 1e-30
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    got = _gemm(gpulib, 1, Ad, Bd, torch.ones(100, 70, dtype=torch.float64, device="cuda"))
    assert bool((got == 0.0).all())
