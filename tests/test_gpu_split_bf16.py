"""The split of FP64 into BF16 hi + lo: each the nearest (ties to even) to x and
to x - hi, in every layout and store width, at halfway cases and at the ends of
the exponent range that takes the integer path -- bit for bit."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _nearest8(x):
    """x rounded to 8 significant bits, ties to even (np.rint), exactly."""
    _, e = np.frexp(x)
    s = np.ldexp(1.0, np.where(x == 0, 0, e - 8))
    return np.rint(x / s) * s


def _values(n, rng):
    x = rng.standard_normal(n) * 10.0 ** rng.uniform(-8, 8, n)
    i = np.arange(n)
    tie = 1.0 + rng.integers(0, 128, n) / 128.0 + rng.choice([-1, 1], n) / 256.0   # halfway for hi
    near = tie + rng.choice([-1, 0, 1], n) * 2.0 ** -rng.integers(17, 50, n)       # and for lo
    x = np.where(i % 3 == 1, near, x)
    x[i % 17 == 0] = 0.0
    x[i % 101 == 5] *= 2.0 ** -60
    x[i % 103 == 7] *= 2.0 ** 90
    return x


@pytest.mark.parametrize("layout", ["rows", "transposed"])
@pytest.mark.parametrize("k", [1, 2, 63, 64, 66, 257, 1026])
@pytest.mark.parametrize("shift", [0, 1])   # elements by which the outputs start off a 4-byte boundary
def test_split_is_nearest(gpulib, layout, k, shift):
    from fricc_gb300 import _lib as L
    rng = np.random.default_rng(1000 * k + shift)
    rows, kp = 70, (3 * k + 7) // 8 * 8
    x = _values(rows * k, rng).reshape(rows, k)
    src = torch.from_numpy(np.ascontiguousarray(x if layout == "rows" else x.T)).cuda()
    ri, sro, sri, sk = (1, k, k, 1) if layout == "rows" else (rows, 0, 1, rows)
    out = [torch.full((rows * kp + 1,), 0x7fff, dtype=torch.int16, device="cuda") for _ in range(2)]
    pa, pb = (ctypes.c_void_p(t.data_ptr() + 2 * shift) for t in out)
    L.check(gpulib.fricc_split_bf16x3_strided(ctypes.c_void_p(src.data_ptr()), rows, k, ri, sro, sri, sk, kp, pa, pb,
                                              L.cur_stream()))
    hi = _nearest8(x)
    lo = _nearest8(x - hi)
    bits = lambda v: torch.from_numpy(v).to(torch.float32).to(torch.bfloat16).view(torch.int16).numpy()  # noqa: E731
    hi, lo = bits(hi), bits(lo)
    pad = np.zeros((rows, kp - 3 * k), dtype=np.int16)
    for t, want in zip(out, (np.hstack([hi, hi, lo, pad]), np.hstack([hi, lo, hi, pad]))):
        got = t.cpu().numpy()[shift:shift + rows * kp].reshape(rows, kp)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("p,q", [((0, 5), (5, 36)), ((0, 5), (5, 37)), ((5, 38), (5, 38)), ((2, 3), (1, 34)), ((0, 0), (0, 33))])
@pytest.mark.parametrize("flip", [False, True])
def test_factor_slices_read_in_place(gpulib, p, q, flip):
    """split_factor of a factor's slices -- rows too short for the transposing
    pass, just long enough, offset, empty, or with transposed orbitals --
    against the split of a copy."""
    from fricc_gb300.cholesky import split_bf16x3, split_factor
    rng = np.random.default_rng(p[1] + q[1])
    L = torch.from_numpy(rng.standard_normal((19, 40, 40))).cuda()
    X = L[:, p[0]:p[1], q[0]:q[1]]
    if flip:
        X = L.transpose(1, 2)[:, p[0]:p[1], q[0]:q[1]]
    if X.numel() == 0:  # refused as the copy's split is
        for f in (split_factor, lambda x: split_bf16x3(x.reshape(x.shape[0], -1).t().contiguous())):
            with pytest.raises(ValueError):
                f(X)
        return
    want = split_bf16x3(X.reshape(X.shape[0], -1).t().contiguous())
    got = split_factor(X)
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    assert torch.equal(split_factor(X, want_b=False).view(torch.int16), want[0].view(torch.int16))
    assert torch.equal(split_factor(X, want_a=False).view(torch.int16), want[1].view(torch.int16))
