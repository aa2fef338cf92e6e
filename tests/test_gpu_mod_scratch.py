"""The modular products under a bound on their scratch: pieces give the bits
of the whole, and with no scratch at all the FP64 and sparse kernels run."""
import ctypes

import pytest
import torch

from test_gpu_mod import _gemm, forced

pytestmark = pytest.mark.gpu


class scratch:
    """fricc_mod_scratch for a block."""

    def __init__(self, lib, nbytes):
        self.lib, self.nbytes = lib, nbytes

    def __enter__(self):
        assert self.lib.fricc_mod_scratch(self.nbytes) == 0

    def __exit__(self, *exc):
        assert self.lib.fricc_mod_scratch(-1) == 0


def _rand(*shape):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(len(shape) + shape[-1]),
                       device="cuda", dtype=torch.float64)


@pytest.mark.parametrize("M,N,K", [(700, 900, 130), (900, 700, 130), (517, 513, 700), (40, 1100, 300)])
@pytest.mark.parametrize("form", ["plain", "transposed", "batch_a", "batch_b"])
def test_panels(gpulib, form, M, N, K):
    """Panels of either operand, ragged last ones, rows of two levels."""
    if form == "plain":
        A, B, C = _rand(M, K), _rand(K, N), _rand(M, N)
    elif form == "transposed":
        A, B, C = _rand(K, M).T, _rand(N, K).T, _rand(N, M).T
    elif form == "batch_a":
        A, B, C = _rand(2, M, K), _rand(K, N).unsqueeze(0).expand(2, K, N), _rand(2, M, N)
    else:
        A, B, C = _rand(M, K).unsqueeze(0).expand(2, M, K), _rand(2, N, K).transpose(1, 2), _rand(2, M, N)
    ref = _gemm(gpulib, 1, A, B, C, -0.5, 1.0)
    with scratch(gpulib, 1 << 20):
        assert torch.equal(_gemm(gpulib, 1, A, B, C, -0.5, 1.0), ref)


@pytest.mark.parametrize("which", ["A", "B", "AB"])
def test_panels_beside_a_prepared_operand(gpulib, which):
    from fricc_gb300 import rccsd_dense as D
    M, N, K = 900, 800, 130
    A, B, C = _rand(M, K), _rand(K, N), _rand(M, N)
    ref = _gemm(gpulib, 1, A, B, C, 1.0, 1.0)
    Am = D.mod_operand(A, M, K, K, 1) if "A" in which else None
    Bm = D.mod_operand(B, N, K, 1, N) if "B" in which else None
    with scratch(gpulib, 1 << 20), forced(gpulib, 1):
        assert torch.equal(D.gemm_f64(A, B, C.clone(), 1.0, 1.0, Am, Bm), ref)


@pytest.mark.parametrize("M,N,K", [(150, 33, 259), (700, 600, 70)])
@pytest.mark.parametrize("nbytes", [1, 1 << 20, 3 << 20, 5 << 20])
def test_replicas_in_groups(gpulib, M, N, K, nbytes):
    """Groups of one (in panels at the larger size), of several and a ragged last one."""
    A, B, C = _rand(5, M, K), _rand(5, K, N), _rand(5, M, N)
    ref = _gemm(gpulib, 1, A, B, C, 1.0, 1.0)
    with scratch(gpulib, nbytes):
        assert torch.equal(_gemm(gpulib, 1, A, B, C, 1.0, 1.0), ref)


def test_no_scratch_leaves_the_other_kernels(gpulib):
    """GEMMs, the eleven terms' entry, fricc_spmm and the batch's."""
    from fricc_gb300 import _lib as L
    from fricc_gb300 import py_rccsd
    vp = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    A, B, C = _rand(90, 70), _rand(70, 80), _rand(90, 80)
    o, v, m, R = 4, 10, 300, 2
    dims, st = L.i64arr((o, o, v, v)), L.cur_stream()
    t2 = _rand(R, o, o, v, v)
    rn = torch.full((R, 2), 0.3, dtype=torch.float64, device="cuda")
    T = py_rccsd.SparseTensor4d(t2[0], t2[0].shape, m, "fri", "systematic", rn=0.3)
    W4, W, out4 = _rand(v, v, v, v), _rand(v * v, 37), _rand(o, o, v, v)
    spb = ctypes.c_void_p()
    L.check(gpulib.fricc_spb_create(R, dims, m, st, ctypes.byref(spb)))
    L.check(gpulib.fricc_spb_recompress_pair(spb, vp(t2), vp(rn), st))

    def all_of(mode):
        res = [_gemm(gpulib, mode, A, B, C, 2.0, 1.0), out4.clone(),
               torch.zeros(o * o, 37, dtype=torch.float64, device="cuda"),
               torch.zeros(R, o * o, 37, dtype=torch.float64, device="cuda")]
        with forced(gpulib, mode):
            py_rccsd.contract_DTSpT(W4, T, res[1], "2323")
            L.check(gpulib.fricc_spmm(T._h, 0, 1, 2, 3, 0.5, vp(W), 37, vp(res[2]), st))
            L.check(gpulib.fricc_spb_spmm(spb, 0, 0, 1, 2, 3, 0.5, vp(W), 0, 37, vp(res[3]), o * o * 37, st))
        return res
    try:
        ref = all_of(0)
        with scratch(gpulib, 0):
            got = all_of(1)
        for x, y in zip(got, ref):
            assert torch.equal(x, y)
    finally:
        gpulib.fricc_spb_destroy(spb)


def test_bound_is_checked(gpulib):
    assert gpulib.fricc_mod_scratch(-2) == 1
    assert gpulib.fricc_mod_scratch(1 << 40) == 0 and gpulib.fricc_mod_scratch(-1) == 0
