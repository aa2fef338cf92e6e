"""The sequential sum where it crosses binades: chunks (4096 addends) cut at the
crossings, more crossings than a chunk's 64 pieces, more such chunks than the 32
with pieces, addends that land on a binade's edge, and long chains -- bit for
bit numpy's left-to-right running sum."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CH, LONG = 4096, 1024 * 4096   # elements of a chunk; chunks the walk's threads take one each


def _addends(name):
    rng = np.random.default_rng(len(name))
    if name == "doubling":            # 60 crossings by single steps
        return np.concatenate([2.0 ** np.arange(-30, 30), rng.random(5000)])
    if name == "many_crossings":      # more than a chunk's pieces
        return 1.3 ** np.arange(900.0)
    if name == "on_the_edge":         # every power of two is hit exactly
        return np.concatenate([np.ones(CH + 7), np.full(3 * CH, 0.5)])
    if name == "near_an_edge":        # a long stay within the slack of 2^20
        return np.concatenate([[2.0 ** 20 - 2.0 ** -20], np.full(9000, 2.0 ** -32), rng.random(9000)])
    if name == "ties":                # halves of a unit, odd and even
        return np.concatenate([[2.0 ** 52 - 3000], np.full(2 * CH, 0.5), np.full(2 * CH, 1.5)])
    if name.startswith("growing"):    # each of that many chunks doubles the sum
        return 2.0 ** (np.arange(float(int(name[7:]) * CH)) / CH) * rng.random(int(name[7:]) * CH)
    if name == "leading_zeros":
        return np.concatenate([np.zeros(CH + 100), rng.random(6000) * 1e-9, np.zeros(50), rng.random(6000)])
    if name == "subnormal":
        return np.concatenate([rng.integers(0, 4, 5000) * 5e-324, rng.random(3000) * 1e-307])
    if name == "to_infinity":
        return np.concatenate([rng.random(5000) * 1e304, np.full(CH, 1e305), rng.random(100)])
    if name == "nan":
        x = rng.random(3 * CH)
        x[CH + 5] = np.nan
        return x
    if name.startswith("len"):
        return rng.random(int(name[3:])) ** 8
    raise KeyError(name)


@pytest.mark.parametrize("name", ["doubling", "many_crossings", "on_the_edge", "near_an_edge", "ties",
                                  "leading_zeros", "growing20", "growing45", "growing100", "subnormal", "to_infinity",
                                  "nan", "len1", "len7", f"len{CH - 1}", f"len{CH + 1}", f"len{LONG}", f"len{LONG + 1}"])
def test_sum_across_binades(gpulib, name):
    from fricc_gb300 import _lib
    x = np.ascontiguousarray(_addends(name))
    with np.errstate(all="ignore"):
        ref = np.add.accumulate(x)
    xd = torch.from_numpy(x).cuda()
    out = torch.empty_like(xd)
    _lib.check(gpulib.fricc_seq_cumsum(ctypes.c_void_p(xd.data_ptr()), xd.numel(), ctypes.c_void_p(out.data_ptr()),
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = out.cpu().numpy()
    nan = np.isnan(ref)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(ref[~nan].view(np.int64), got[~nan].view(np.int64))
