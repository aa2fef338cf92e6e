"""The pivotal sampler's weight walk in parallel segments, where it can go
wrong: region edges, long stretches without a wrap, sums that land on powers
of two and ties, probabilities of exactly 1: bit for bit the oracle's."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tensor(name, rng):
    if name.startswith("n"):           # sizes around the region length and its multiples
        n = int(name[1:])
        return rng.standard_normal(n) * rng.random(n), max(1, n // 9)
    if name == "sparse":               # regions without a wrap
        x = np.zeros(60_000)
        x[rng.choice(60_000, 400, replace=False)] = rng.random(400) + 0.5
        return x, 100
    if name == "gap":                  # a long run of zeros between two dense parts
        x = np.concatenate([rng.random(5000), np.zeros(40_000), rng.random(5000)])
        return x, 900
    if name == "quarter":              # every sum a multiple of 1/4: the weight hits 1 exactly
        return np.full(40_000, 0.5), 10_000
    if name == "tenth":                # ten tenths round below 1: the fixed-point prediction is off at every wrap
        return np.full(40_000, 0.5), 4000
    if name == "dyadic":               # probabilities with few bits: ties at the wraps
        return rng.integers(1, 16, 50_000) / 16.0, 8192
    if name == "half_ulp":             # probabilities whose last bit is half an ulp of the wrap's sum
        return (1.0 + rng.integers(0, 2, 50_000) * 2.0 ** -50) * rng.integers(1, 9, 50_000), 6000
    if name == "ones":                 # most probabilities near or at 1
        return np.concatenate([np.full(3000, 1.0), rng.random(20_000) * 1e-3]), 2999
    if name == "large":
        return rng.standard_normal(1_500_000) * np.exp(rng.standard_normal(1_500_000)), 90_000
    raise KeyError(name)


@pytest.mark.parametrize("name", ["n1", "n2", "n127", "n128", "n129", "n255", "n257", "n1000", "sparse", "gap", "quarter",
                                  "tenth", "dyadic", "half_ulp", "ones", "large"])
def test_walk_vs_oracle(gpulib, oracle, name):
    from fricc_gb300 import _lib as L
    from fricc_gb300.rng import GlibcRand
    rng = np.random.default_rng(len(name) + 40)
    x, m = _tensor(name, rng)
    x = np.ascontiguousarray(x)
    n = x.size
    st = L.cur_stream()
    draws = torch.empty(n, dtype=torch.float64, device="cuda")
    h, _ = L.hist_arg(GlibcRand(7))
    L.check(gpulib.fricc_glibc_uniforms(h, n, ctypes.c_void_p(draws.data_ptr()), st))
    xd = torch.from_numpy(x).cuda()
    flat = torch.empty(m, dtype=torch.int64, device="cuda")
    vals = torch.empty(m, dtype=torch.float64, device="cuda")
    nd, used = ctypes.c_int64(0), ctypes.c_int64(0)
    h, _ = L.hist_arg(GlibcRand(7))
    rc = gpulib.fricc_compress_pivotal(ctypes.c_void_p(xd.data_ptr()), n, m, h, ctypes.c_void_p(flat.data_ptr()),
                                       ctypes.c_void_p(vals.data_ptr()), ctypes.byref(nd), ctypes.byref(used), st)
    try:
        oi, ov, ond, oused = oracle.fri_compression_pivotal(x, m, draws=draws.cpu().numpy())
    except Exception:
        assert rc == 8 or rc == 3   # the oracle's own exits: FRICC_ERR_PIVOTAL, FRICC_ERR_P_GT_ONE
        return
    L.check(rc)
    assert used.value == oused and nd.value == ond
    np.testing.assert_array_equal(flat.cpu().numpy(), oi)
    assert np.array_equal(vals.cpu().numpy().view(np.int64), ov.view(np.int64))
