"""Samples of one compression that fall on the same element: every one of
them reaches the zero-filled operand of the modular products."""
import pytest
import torch

from test_gpu_mod import forced

pytestmark = pytest.mark.gpu


def test_two_samples_of_one_element(gpulib):
    """With a remaining norm at or below 1e-14 nothing is kept whole, a
    probability can be 1, and where the partial sums cross a power of two
    its interval can hold two samples: here elements 4 (twice) and 3 (none)."""
    from fricc_gb300 import py_rccsd
    u = 2.0 ** -53
    p = [1.0, 1.0, 1.0, 1.0 - 2.0 ** -51, 1.0, 1.0, 1.0, 1.0]
    x = torch.zeros(2, 2, 3, 3, dtype=torch.float64, device="cuda")
    x.view(-1)[:8] = torch.tensor(p, dtype=torch.float64) * u
    T = py_rccsd.SparseTensor4d(x, x.shape, 8, "fri", "systematic", rn=1.0 - 2.0 ** -51 - 2.0 ** -53)
    idx = [T.get_element(k)[0] for k in range(8)]
    flat = sorted(((i[0] * 2 + i[1]) * 3 + i[2]) * 3 + i[3] for i in idx)
    assert flat == [0, 1, 2, 4, 4, 5, 6, 7]
    g = torch.Generator(device="cuda").manual_seed(1)
    W = torch.randn(3, 3, 3, 3, generator=g, device="cuda", dtype=torch.float64)
    res = []
    for f in (0, 1):
        with forced(gpulib, f):
            out = torch.zeros(2, 2, 3, 3, dtype=torch.float64, device="cuda")
            py_rccsd.contract_DTSpT(W, T, out, "2323")
            res.append(out)
    assert float((res[0] - res[1]).abs().max()) <= 1e-14 * float(res[0].abs().max())


def test_absent_and_stored_zeros(gpulib):
    """A kept element that is zero multiplies a NaN (also at index 0); an
    absent one does not."""
    from fricc_gb300 import py_rccsd
    x = torch.zeros(2, 2, 3, 3, dtype=torch.float64, device="cuda")
    x[1, 0, 2, 1] = 1.0
    T = py_rccsd.SparseTensor4d(x, x.shape, 3, "largest", "systematic")  # with the zeros at 0 and 1
    W = torch.ones(3, 3, 3, 3, dtype=torch.float64, device="cuda")
    W[0, 0, 0, 0] = float("nan")  # the key of the zero kept at index 0
    W[1, 1, 1, 1] = float("nan")  # a key no kept element has
    res = []
    for f in (0, 1):
        with forced(gpulib, f):
            out = torch.zeros(2, 2, 3, 3, dtype=torch.float64, device="cuda")
            py_rccsd.contract_DTSpT(W, T, out, "2323")
            res.append(out)
    assert int(torch.isnan(res[0]).sum()) == 1 and bool(torch.isnan(res[0][0, 0, 0, 0]))
    assert torch.equal(torch.isnan(res[0]), torch.isnan(res[1]))
