"""Compressions that take each route of the candidate sort (direct ranking,
cooperative digit passes) and of the remaining-norm chain (its first chunks
in one block, the general chain), at the routes' limits: bit for bit the
oracle's, and a batch's replicas bit for bit their single calls'."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

RANK_MAX, FIRST = 16384, 8 * 4096  # candidates ranked directly; chain elements of the first block


def _inputs(name):
    rng = np.random.default_rng(len(name))
    if name == "long_d":              # |D| far past the first chunks, more candidates than are ranked
        return 2.0 ** (-np.arange(60_000) / 4000.0) * rng.choice([-1.0, 1.0], 60_000), 50_000
    if name == "d_at_first":          # |D| at the end of the first chunks
        x = np.concatenate([np.full(FIRST, 1.0), np.full(30_000, 1e-9)])
        return rng.permutation(x), FIRST + 500
    if name == "d_past_first":
        x = np.concatenate([np.full(FIRST + 1, 1.0), np.full(30_000, 1e-9)])
        return rng.permutation(x), FIRST + 500
    if name == "ties_at_rank":        # equal keys on both sides of the ranking limit
        return np.concatenate([np.full(RANK_MAX + 1, 0.5), rng.random(9000) * 0.1]), 17_000
    if name == "no_d":                # nothing passes the acceptance test
        return np.full(30_000, 0.25), 300
    if name == "inf_top":
        x = rng.standard_normal(30_000)
        x[[5, 700]] = np.inf, -np.inf
        return x, 4000
    if name == "nan":
        x = rng.standard_normal(30_000)
        x[12_345] = np.nan
        return x, 4000
    if name == "tiny":                # every magnitude subnormal
        return rng.standard_normal(30_000) * 5e-324 * 1e5, 4000
    if name == "huge":                # one_norm overflows to infinity
        return rng.standard_normal(30_000) * 1e308, 4000
    raise KeyError(name)


def _same(a, b):
    na, nb = np.isnan(a), np.isnan(b)
    return np.array_equal(na, nb) and np.array_equal(a[~na].view(np.int64), b[~nb].view(np.int64))


@pytest.mark.parametrize("name", ["long_d", "d_at_first", "d_past_first", "ties_at_rank", "no_d", "inf_top", "nan",
                                  "tiny", "huge"])
def test_routes_vs_oracle(gpulib, oracle, name):
    from fricc_gb300 import py_rccsd
    x, m = _inputs(name)
    x = np.ascontiguousarray(x).reshape(1, 1, 1, -1)
    for kind in ("fri", "largest"):
        if name == "nan" and kind == "largest":
            continue  # the oracle's order of a NaN against the rest is not defined
        with np.errstate(all="ignore"):
            ref = oracle.SparseTensor4d(x, x.shape, m, kind, "systematic", rn=0.37)
        t = py_rccsd.SparseTensor4d(x, x.shape, m, kind, "systematic", rn=0.37 if kind == "fri" else 0.0)
        flat, vals = t.export()
        np.testing.assert_array_equal(flat, ref.flat, err_msg=kind)
        assert _same(vals, ref.vals), kind


@pytest.mark.parametrize("n", [RANK_MAX - 1, RANK_MAX, RANK_MAX + 1, 3 * RANK_MAX + 7])
def test_largest_sorts_all(gpulib, n):
    """Every element a candidate, around the ranking limit: the stable
    descending order (exact: indices and bits)."""
    from fricc_gb300 import py_rccsd
    rng = np.random.default_rng(n)
    x = np.round(rng.standard_normal(n) * 500) / 500.0
    t = py_rccsd.SparseTensor4d(x.reshape(1, 1, 1, n), (1, 1, 1, n), n, "largest")
    flat, vals = t.export()
    order = np.argsort(-np.abs(x), kind="stable")
    np.testing.assert_array_equal(flat, order)
    assert _same(vals, x[order])


def test_batch_mixes_routes(gpulib):
    """Replicas of one batch on different routes: each as its paired call."""
    from fricc_gb300 import _lib as L
    names = ["long_d", "no_d", "ties_at_rank"]
    n, m = 25_000, 17_500
    xs = []
    for nm in names:
        x, _ = _inputs(nm)
        xs.append(np.resize(x, n))
    x = torch.from_numpy(np.stack(xs)).cuda()
    R, dims = len(names), L.i64arr((1, 1, 1, n))
    st = L.cur_stream()
    rn = torch.tensor([[0.1 + 0.2 * r, 0.9 - 0.2 * r] for r in range(R)], dtype=torch.float64, device="cuda")
    spb = ctypes.c_void_p()
    L.check(gpulib.fricc_spb_create(R, dims, m, st, ctypes.byref(spb)))
    try:
        vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        L.check(gpulib.fricc_spb_recompress_pair(spb, vp(x), vp(rn), st))
        for r in range(R):
            for which in (0, 1):
                h = ctypes.c_void_p()
                L.check(gpulib.fricc_sp_create(vp(x[r]), dims, m, 0, 0, float(rn[r, which]), st, ctypes.byref(h)))
                got, ref = [], []
                for fn, head, into in ((gpulib.fricc_spb_export, (spb, which, r), got),
                                       (gpulib.fricc_sp_export, (h,), ref)):
                    flat, vals = np.empty(m, dtype=np.int64), np.empty(m)
                    L.check(fn(*head, ctypes.c_void_p(flat.ctypes.data), ctypes.c_void_p(vals.ctypes.data), st))
                    into += [flat, vals]
                L.check(gpulib.fricc_sp_destroy(h))
                np.testing.assert_array_equal(got[0], ref[0])
                assert _same(got[1], ref[1])
    finally:
        L.check(gpulib.fricc_spb_destroy(spb))
