"""The device's glibc stream where its chunks (248 draws) and the powers of their
jump matrix change: draws and the history handed back, against the Python one."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CH = 31 * 8


@pytest.mark.parametrize("k", [1, 30, CH - 1, CH, CH + 1, 2 * CH, 2 * CH + 1, 4 * CH, 33 * CH - 5, 64 * CH, 64 * CH + 40,
                               257 * CH + 1])
def test_stream_at_chunk_limits(gpulib, k):
    from fricc_gb300 import _lib as L
    from fricc_gb300.rng import GlibcRand
    g, ref = GlibcRand(k), GlibcRand(k)
    want = np.array([ref.uniform() for _ in range(k)])
    out = torch.empty(k, dtype=torch.float64, device="cuda")
    hist, writeback = L.hist_arg(g)
    L.check(gpulib.fricc_glibc_uniforms(hist, k, ctypes.c_void_p(out.data_ptr()), L.cur_stream()))
    writeback()
    assert np.array_equal(out.cpu().numpy(), want)
    assert [g.rand() for _ in range(40)] == [ref.rand() for _ in range(40)]
