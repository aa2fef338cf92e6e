"""The pivotal sampler with few samples, or long stretches without one: the
walk goes to the serial kernel where parallel segments would not pay, with the
oracle's bits and draws on either side of that line."""
import ctypes
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _compress(lib, xd, m, seed=7):
    from fricc_gb300 import _lib as L
    from fricc_gb300.rng import GlibcRand
    flat = torch.empty(m, dtype=torch.int64, device="cuda")
    vals = torch.empty(m, dtype=torch.float64, device="cuda")
    nd, used = ctypes.c_int64(0), ctypes.c_int64(0)
    h, _ = L.hist_arg(GlibcRand(seed))
    L.check(lib.fricc_compress_pivotal(ctypes.c_void_p(xd.data_ptr()), xd.numel(), m, h, ctypes.c_void_p(flat.data_ptr()),
                                       ctypes.c_void_p(vals.data_ptr()), ctypes.byref(nd), ctypes.byref(used),
                                       L.cur_stream()))
    return flat, vals, nd.value, used.value


def _check(lib, oracle, x, m):
    from fricc_gb300 import _lib as L
    from fricc_gb300.rng import GlibcRand
    draws = torch.empty(x.size, dtype=torch.float64, device="cuda")
    h, _ = L.hist_arg(GlibcRand(7))
    L.check(lib.fricc_glibc_uniforms(h, x.size, ctypes.c_void_p(draws.data_ptr()), L.cur_stream()))
    flat, vals, nd, used = _compress(lib, torch.from_numpy(np.ascontiguousarray(x)).cuda(), m)
    oi, ov, ond, oused = oracle.fri_compression_pivotal(x, m, draws=draws.cpu().numpy())
    assert (nd, used) == (ond, oused)
    np.testing.assert_array_equal(flat.cpu().numpy(), oi)
    assert np.array_equal(vals.cpu().numpy().view(np.int64), ov.view(np.int64))


@pytest.mark.parametrize("m", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("n", [300, 40_000])
def test_few_samples(gpulib, oracle, n, m):
    _check(gpulib, oracle, np.random.default_rng(m).random(n) + 0.5, m)


@pytest.mark.parametrize("share", [0.3, 0.46, 0.48, 0.7])
@pytest.mark.parametrize("where", ["front", "middle", "end"])
def test_long_stretches(gpulib, oracle, where, share):
    """Zeros over a share of the tensor on both sides of the line (15/32)."""
    rng = np.random.default_rng(int(100 * share))
    n = 50_000
    x, z = rng.random(n) + 0.5, int(n * share)
    at = {"front": 0, "middle": (n - z) // 2, "end": n - z}[where]
    x[at:at + z] = 0.0
    _check(gpulib, oracle, x, 900)


def test_one_sample_is_not_walked_twice(gpulib):
    """One sample leaves one segment: it used to take three times as long as
    three samples, whose segments run side by side (155 and 52 ms)."""
    x = torch.rand(200_000, generator=torch.Generator(device="cuda").manual_seed(1), device="cuda",
                   dtype=torch.float64) + 0.5
    best = {}
    for m in (1, 3):
        for _ in range(4):
            torch.cuda.synchronize()
            t = time.perf_counter()
            _compress(gpulib, x, m)
            torch.cuda.synchronize()
            best[m] = min(best.get(m, 1e9), time.perf_counter() - t)
    assert best[1] < 2.0 * best[3], best
