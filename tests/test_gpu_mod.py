"""The modular tensor-core products (FP64 accuracy on tcgen05) against exact
sums and against the FP64 kernels, over tile edges, strides, batches,
magnitudes and the routes they replace."""
import ctypes
import math

import numpy as np
import pytest
import torch

from conftest import REPO  # noqa: F401

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


class forced:
    """fricc_mod_select for a block: 0 the FP64 kernels, 1 the modular products."""

    def __init__(self, lib, value):
        self.lib, self.value = lib, value

    def __enter__(self):
        assert self.lib.fricc_mod_select(self.value) == 0

    def __exit__(self, *exc):
        assert self.lib.fricc_mod_select(-1) == 0


def _gemm(lib, force, A, B, C, alpha=1.0, beta=0.0):
    from fricc_gb300 import rccsd_dense as D
    out = C.clone(memory_format=torch.preserve_format)
    out = torch.empty_strided(C.shape, C.stride(), dtype=C.dtype, device=C.device).copy_(C)
    with forced(lib, force):
        D.gemm_f64(A, B, out, alpha, beta)
    return out


def _exact(A, B):
    """A @ B to far beyond FP64, as (hi, lo): per-element two-products summed by math.fsum."""
    M, K = A.shape
    N = B.shape[1]
    R = np.empty((M, N))
    split = 134217729.0
    for i in range(M):
        a = A[i][:, None]
        p = a * B
        ah = a * split - (a * split - a)
        bh = B * split - (B * split - B)
        al, bl = a - ah, B - bh
        e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
        for j in range(N):
            R[i, j] = math.fsum(np.concatenate([p[:, j], e[:, j]]).tolist())
    return R


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (5, 7, 3), (127, 31, 255), (128, 32, 256), (129, 33, 257), (130, 300, 64),
                                   (257, 65, 511), (64, 513, 513), (5, 520, 1030), (300, 6, 2000)])
def test_integers_exact(gpulib, M, N, K):
    """Integer matrices whose products stay below 2^53: bit for bit."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randint(-2 ** 19, 2 ** 19, (M, K), generator=g, device="cuda").double()
    B = torch.randint(-2 ** 19, 2 ** 19, (K, N), generator=g, device="cuda").double()
    C = torch.zeros(M, N, dtype=torch.float64, device="cuda")
    got = _gemm(gpulib, 1, A, B, C)
    ref = (A.cpu().long() @ B.cpu().long()).double()
    assert torch.equal(got.cpu(), ref)


@pytest.mark.parametrize("K", [255, 256, 4096])
def test_largest_residues(gpulib, K):
    """Constant operands: every product of a modulus has the same sign, and
    over the values every residue takes its extremes."""
    for v in (2.0 ** 53 - 1, -(2.0 ** 53 - 1), 6004799503160661.0, 1.0 / 3.0):
        A = torch.full((130, K), v, dtype=torch.float64, device="cuda")
        B = torch.full((K, 40), -v * 0.75, dtype=torch.float64, device="cuda")
        got = _gemm(gpulib, 1, A, B, torch.zeros(130, 40, dtype=torch.float64, device="cuda"))
        ref = math.fsum(_exact(np.full((1, K), v), np.full((K, 1), -v * 0.75)).ravel())
        assert float((got - ref).abs().max()) <= 2 * U * abs(ref)


@pytest.mark.parametrize("M,N,K", [(40, 36, 30), (33, 48, 150), (40, 40, 900), (24, 20, 6000)])
def test_error_no_larger_than_fp64(gpulib, M, N, K):
    """Against sums exact to FP64: the error (2-norm) is at most that of
    the FP64 kernel plus a final rounding of both."""
    rng = np.random.default_rng(K)
    A = rng.standard_normal((M, K)) * np.exp(rng.standard_normal((M, K)))
    B = rng.standard_normal((K, N)) * np.exp(rng.standard_normal((K, N)))
    A[:, rng.random(K) < 0.3] = 0.0
    ref = _exact(A, B)
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    C = torch.zeros(M, N, dtype=torch.float64, device="cuda")
    err = [np.linalg.norm(_gemm(gpulib, f, Ad, Bd, C).cpu().numpy() - ref) / np.linalg.norm(ref) for f in (0, 1)]
    assert err[1] <= max(err[0], U), err


def _bound(A, B):
    """A componentwise bound for either kernel: a sum in any order."""
    K = A.shape[-1]
    return (K + 8) * U * (A.abs() @ B.abs())


@pytest.mark.parametrize("kind", ["scales", "orthogonal", "zeros", "subnormal", "spike", "overflow"])
def test_magnitudes_componentwise(gpulib, kind):
    """Inputs far from one scale keep FP64's componentwise bound (by the
    check of every output and the FP64 recomputation behind it)."""
    rng = np.random.default_rng(5)
    A, B = rng.standard_normal((70, 200)), rng.standard_normal((200, 90))
    if kind == "scales":        # rows and columns over the whole exponent range
        A *= 10.0 ** rng.integers(-140, 140, (70, 1))
        B *= 10.0 ** rng.integers(-140, 140, (1, 90))
    elif kind == "orthogonal":  # the large elements of A meet the small ones of B
        A[:, ::2] *= 1e-12
        B[1::2] *= 1e-12
    elif kind == "zeros":
        A[rng.random(A.shape) < 0.9] = 0.0
        A[3], B[:, 7] = 0.0, 0.0
    elif kind == "subnormal":
        A[:20] *= 1e-310
        B[:, :20] *= 1e-200
    elif kind == "spike":
        A[np.arange(70), rng.integers(0, 200, 70)] = 1e15
        B[5] = 0.0
    else:
        A *= 1e200
        B *= 1e150
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    C = torch.zeros(70, 90, dtype=torch.float64, device="cuda")
    got, ref = _gemm(gpulib, 1, Ad, Bd, C), _gemm(gpulib, 0, Ad, Bd, C)
    fin = torch.isfinite(ref)
    assert torch.equal(fin, torch.isfinite(got))
    tol = 2 * _bound(Ad, Bd) + 2e-323
    assert bool(((got - ref).abs()[fin] <= tol[fin]).all())


def test_nonfinite_rows(gpulib):
    rng = np.random.default_rng(6)
    A, B = rng.standard_normal((150, 64)), rng.standard_normal((64, 50))
    A[3, 5], A[77, 0], B[9, 11] = np.nan, np.inf, -np.inf
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    C = torch.zeros(150, 50, dtype=torch.float64, device="cuda")
    got, ref = _gemm(gpulib, 1, Ad, Bd, C).cpu(), _gemm(gpulib, 0, Ad, Bd, C).cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isinf(got), torch.isinf(ref))
    assert float((got - ref)[fin].abs().max()) <= 1e-13


def _views(form, M, N, K, g):
    def r(*s):
        return torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)
    b = 3
    if form == "plain":
        return r(M, K), r(K, N), r(M, N)
    if form == "transposed":
        return r(K, M).T, r(N, K).T, r(N, M).T
    if form == "sliced":
        return r(M, 2 * K + 1)[:, 1::2], r(K + 3, N + 5)[3:, 5:], r(M, 3 * N)[:, ::3]
    if form == "batch_a":
        return r(b, M, K), r(K, N).unsqueeze(0).expand(b, K, N), r(b, M, N)
    if form == "batch_b":
        return r(M, K).unsqueeze(0).expand(b, M, K), r(b, N, K).transpose(1, 2), r(b, M, N)
    if form == "batch_ab":
        return r(b, M, K), r(b, K, N), r(b, N, M).transpose(1, 2)
    if form == "b2_ab":
        return r(2, b, M, K), r(2, b, K, N), r(2, b, M, N)
    if form == "b2_a_b1":      # A moves with the inner level, B with the outer one
        return r(1, b, M, K).expand(2, b, M, K), r(2, 1, K, N).expand(2, b, K, N), r(2, b, M, N)
    if form == "b2_rep_inner":  # the inner level moves both, the outer one only A
        return r(2, b, M, K), r(1, b, K, N).expand(2, b, K, N), r(2, b, M, N)
    raise KeyError(form)


@pytest.mark.parametrize("form", ["plain", "transposed", "sliced", "batch_a", "batch_b", "batch_ab", "b2_ab", "b2_a_b1",
                                  "b2_rep_inner"])
@pytest.mark.parametrize("alpha,beta", [(1.0, 0.0), (-1.0, 1.0), (0.5, -2.0)])
def test_gemm_forms(gpulib, form, alpha, beta):
    """Every stride and batch form the GEMMs take: as the FP64 kernel."""
    for M, N, K in ((9, 70, 40), (150, 33, 259)):
        g = torch.Generator(device="cuda").manual_seed(M)
        A, B, C = _views(form, M, N, K, g)
        got, ref = (_gemm(gpulib, f, A, B, C, alpha, beta) for f in (1, 0))
        scale = _bound(A, B).max() * abs(alpha) + 4 * U * C.abs().max() * abs(beta)
        assert float((got - ref).abs().max()) <= float(scale)


def test_split_k_and_panels(gpulib):
    """A long K with few tiles (split K) and reps of one shape: the replicas bit for bit the lone products."""
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.randn(4, 20, 40_000, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(4, 40_000, 30, generator=g, device="cuda", dtype=torch.float64)
    C = torch.zeros(4, 20, 30, dtype=torch.float64, device="cuda")
    got = _gemm(gpulib, 1, A, B, C)
    for r in range(4):
        assert torch.equal(got[r], _gemm(gpulib, 1, A[r], B[r], C[r]))
    ref = _gemm(gpulib, 0, A, B, C)
    assert float((got - ref).abs().max()) <= float(_bound(A, B).max())


def test_prepared_operands(gpulib):
    from fricc_gb300 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(2)
    A = torch.randn(300, 77, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(77, 45, generator=g, device="cuda", dtype=torch.float64)
    C = torch.randn(300, 45, generator=g, device="cuda", dtype=torch.float64)
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731

    def prep(x, rows, k, rs, ks):
        buf = torch.empty(gpulib.fricc_mod_bytes(rows, k), dtype=torch.uint8, device="cuda")
        L.check(gpulib.fricc_mod_prepare(vp(x), rows, k, rs, ks, vp(buf), L.cur_stream()))
        return buf
    Am, Bm = prep(A, 300, 77, 77, 1), prep(B, 45, 77, 1, 45)
    ref = _gemm(gpulib, 1, A, B, C, 1.0, 1.0)
    with forced(gpulib, 1):
        for a, b in ((Am, None), (None, Bm), (Am, Bm)):
            out = C.clone()
            L.check(gpulib.fricc_gemm_f64_mod(vp(A), vp(a) if a is not None else None, vp(B),
                                              vp(b) if b is not None else None, vp(out), 1, 1, 300, 45, 77,
                                              L.i64arr((77, 1, 0, 0)), L.i64arr((45, 1, 0, 0)), L.i64arr((45, 1, 0, 0)),
                                              1.0, 1.0, L.cur_stream()))
            assert torch.equal(out, ref)


@pytest.mark.parametrize("o,v,frac", [(3, 7, 0.3), (5, 16, 0.1), (8, 33, 0.05)])
def test_terms_vs_sparse_kernel(gpulib, o, v, frac):
    """The eleven terms, contiguous and strided W and out, on a FRI-compressed T."""
    from fricc_gb300 import py_rccsd
    rng = np.random.default_rng(o)
    t2 = torch.from_numpy(rng.standard_normal((o, o, v, v)) * rng.random((o, o, v, v)) ** 3).cuda()
    T = py_rccsd.SparseTensor4d(t2, t2.shape, max(4, int(t2.numel() * frac)), "fri", "systematic", rn=0.4)
    d = {"o": o, "v": v}
    shapes = {"0101": ("oooo", "oovv"), "2323": ("vvvv", "oovv"), "1302": ("voov", "oovv"), "1202": ("vovo", "oovv"),
              "1303": ("voov", "oovv"), "1203": ("vovo", "oovv"), "1323": ("ovov", "oooo"), "0112": ("ovov", "voov"),
              "0113": ("ovov", "voov"), "0313": ("ovov", "voov"), "0312": ("ovov", "vovo")}
    for term, (ws, os_) in shapes.items():
        for perm in ((0, 1, 2, 3), (3, 2, 1, 0), (1, 3, 0, 2), (2, 0, 3, 1)):
            inv = [perm.index(k) for k in range(4)]
            def make(sh):
                sz = [d[c] for c in sh]
                return torch.from_numpy(rng.standard_normal([sz[p] for p in perm])).cuda().permute(inv)
            W, out = make(ws), make(os_)
            res = []
            for f in (0, 1):
                with forced(gpulib, f):
                    x = torch.empty_strided(out.shape, out.stride(), dtype=out.dtype, device="cuda").copy_(out)
                    py_rccsd.contract_DTSpT(W, T, x, term)
                    res.append(x)
            scale = float(res[0].abs().max())
            assert float((res[0] - res[1]).abs().max()) <= 1e-13 * scale, (term, perm)


def test_terms_nan_and_absent(gpulib):
    """A NaN of W reaches only the outputs whose bucket holds its key, and a
    NaN amplitude only its own bucket, as in the sparse kernel; unmatched
    samples (index 0) add up."""
    from fricc_gb300 import py_rccsd
    rng = np.random.default_rng(8)
    o, v = 4, 12
    t2 = np.zeros((o, o, v, v))
    t2.ravel()[rng.choice(t2.size, 200, replace=False)] = rng.standard_normal(200)
    t2[0, 0, 0, 0] = 0.125
    cases = [(t2, 150), (t2, 400)]            # 400 > nonzeros: samples without an interval keep index 0
    for x, m in cases:
        for poison in (False, True):
            xs = torch.from_numpy(x.copy()).cuda()
            T = py_rccsd.SparseTensor4d(xs, xs.shape, m, "largest" if poison else "fri", "systematic", rn=0.3)
            W = torch.from_numpy(rng.standard_normal((v, v, v, v))).cuda()
            if poison:
                W[3, 4, 5, 6], W[1, 1, 1, 1] = float("nan"), float("inf")
            res = []
            for f in (0, 1):
                with forced(gpulib, f):
                    out = torch.zeros(o, o, v, v, dtype=torch.float64, device="cuda")
                    py_rccsd.contract_DTSpT(W, T, out, "2323")
                    res.append(out)
            assert torch.equal(torch.isnan(res[0]), torch.isnan(res[1]))
            assert torch.equal(torch.isinf(res[0]), torch.isinf(res[1]))
            fin = torch.isfinite(res[0])
            if bool(fin.any()):
                scale = float(res[0][fin].abs().max()) or 1.0
                assert float((res[0] - res[1])[fin].abs().max()) <= 1e-12 * scale


def test_batch_terms_match_lone(gpulib):
    """Batched sparse terms (shared and per-replica W): bit for bit the lone calls."""
    from fricc_gb300 import _lib as L
    rng = np.random.default_rng(3)
    R, o, v = 3, 4, 10
    m = 300
    t2 = torch.from_numpy(rng.standard_normal((R, o, o, v, v))).cuda()
    rn = torch.from_numpy(rng.random((R, 2))).cuda()
    dims, st = L.i64arr((o, o, v, v)), L.cur_stream()
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    spb = ctypes.c_void_p()
    L.check(gpulib.fricc_spb_create(R, dims, m, st, ctypes.byref(spb)))
    L.check(gpulib.fricc_spb_recompress_pair(spb, vp(t2), vp(rn), st))
    lone = []
    for r in range(R):
        h = ctypes.c_void_p()
        L.check(gpulib.fricc_sp_create(vp(t2[r]), dims, m, 0, 0, float(rn[r, 0]), st, ctypes.byref(h)))
        lone.append(h)
    try:
        with forced(gpulib, 1):
            for pa, pb, ka, kb, qs in ((0, 1, 2, 3, 37), (1, 3, 0, 2, 40), (2, 3, 0, 1, 16)):
                dd = (o, o, v, v)
                nP, keys = dd[pa] * dd[pb], dd[ka] * dd[kb]
                for shared in (True, False):
                    W = torch.from_numpy(rng.standard_normal((1 if shared else R, keys, qs))).cuda()
                    O0 = torch.from_numpy(rng.standard_normal((R, nP, qs))).cuda()
                    got = O0.clone()
                    L.check(gpulib.fricc_spb_spmm(spb, 0, pa, pb, ka, kb, -0.5, vp(W), 0 if shared else keys * qs, qs,
                                                  vp(got), nP * qs, st))
                    for r in range(R):
                        ref = O0[r].clone()
                        L.check(gpulib.fricc_spmm(lone[r], pa, pb, ka, kb, -0.5, vp(W[0 if shared else r]), qs, vp(ref),
                                                  st))
                        assert torch.equal(got[r], ref)
    finally:
        for h in lone:
            gpulib.fricc_sp_destroy(h)
        gpulib.fricc_spb_destroy(spb)
