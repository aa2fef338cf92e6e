"""The symmetrised accumulation at the edges of its tiles (32 x 32) and pairs
(i <= j), for views of every layout and for replicas: coefficients that are
powers of two make every product exact, so the sums are numpy's bit for bit."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("perm", [(0, 1, 2, 3), (2, 3, 0, 1), (3, 2, 1, 0), (1, 3, 0, 2)])
@pytest.mark.parametrize("o,v", [(1, 1), (1, 33), (2, 31), (5, 32), (7, 65)])
def test_symadd_edges(gpulib, o, v, perm):
    from fricc_gb300 import _lib as L
    rng = np.random.default_rng(o * 100 + v)
    R, shape = 3, (o, o, v, v)
    out = rng.standard_normal((R, *shape))
    Xb = rng.standard_normal((R, *[shape[p] for p in perm]))           # memory order perm
    inv = np.argsort(perm)
    X = Xb.transpose(0, *[1 + k for k in inv])                         # as [r, i, j, a, b]
    for coef in (1.0, -1.0, 0.5):
        want = out + coef * (X + X.transpose(0, 2, 1, 4, 3))
        xd = torch.from_numpy(Xb).cuda().permute(0, *[int(1 + k) for k in inv])
        od = torch.from_numpy(out.copy()).cuda()
        L.check(gpulib.fricc_symadd(ctypes.c_void_p(od.data_ptr()), ctypes.c_void_p(xd.data_ptr()), o, v,
                                    L.i64arr(xd.stride()[1:]), coef, L.cur_stream()))
        np.testing.assert_array_equal(od[0].cpu().numpy(), want[0])
        od = torch.from_numpy(out.copy()).cuda()
        L.check(gpulib.fricc_symadd_b(ctypes.c_void_p(od.data_ptr()), ctypes.c_void_p(xd.data_ptr()), R, o, v,
                                      L.i64arr(xd.stride()), coef, L.cur_stream()))
        np.testing.assert_array_equal(od.cpu().numpy(), want)
