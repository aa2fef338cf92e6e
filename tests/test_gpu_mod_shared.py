"""Products of a batch that neither operand moves along, with operands
prepared once: every product of the batch, from the prepared rows alone."""
import ctypes

import pytest
import torch

from test_gpu_mod import _gemm, forced

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,batch2", [(3, 1), (1, 2), (3, 2)])
@pytest.mark.parametrize("which", ["A", "B", "AB"])
def test_shared_by_the_whole_batch(gpulib, which, batch, batch2):
    from fricc_gb300 import _lib as L
    from fricc_gb300 import rccsd_dense as D
    M, N, K = 150, 40, 77
    g = torch.Generator(device="cuda").manual_seed(batch)
    A = torch.randn(M, K, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(K, N, generator=g, device="cuda", dtype=torch.float64)
    C = torch.randn(batch2, batch, M, N, generator=g, device="cuda", dtype=torch.float64)
    ref = torch.stack([_gemm(gpulib, 1, A, B, c, 1.0, 1.0) for c in C.view(-1, M, N)]).view(C.shape)
    Am = D.mod_operand(A, M, K, K, 1) if "A" in which else None
    Bm = D.mod_operand(B, N, K, 1, N) if "B" in which else None
    vp = lambda t: ctypes.c_void_p(t.data_ptr()) if t is not None else None  # noqa: E731
    with forced(gpulib, 1):
        L.check(gpulib.fricc_gemm_f64_mod(vp(A), vp(Am), vp(B), vp(Bm), vp(C), batch, batch2, M, N, K,
                                          L.i64arr((K, 1, 0, 0)), L.i64arr((N, 1, 0, 0)),
                                          L.i64arr((N, 1, M * N, batch * M * N)), 1.0, 1.0, L.cur_stream()))
    assert torch.equal(C, ref)
