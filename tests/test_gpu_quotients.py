"""The amplitudes' division by the denominators, done on the integer pipe: bit
for bit numpy's, for significands next to powers of two, exact and nearly halfway
quotients, and numbers that take the division instruction."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bits(u):
    return np.asarray(u, dtype=np.uint64).view(np.float64)


def _inputs(name, o, v, rng):
    nov, n = o * v, (o * v) ** 2
    one = np.uint64(0x3ff0000000000000)
    if name == "random":
        eia = -rng.random(nov) * 3 - 0.1
        return rng.standard_normal(n) * 10.0 ** rng.uniform(-9, 2, n), eia
    if name == "edges":       # denominators 2^k (1 + few ulp) or 2^k (2 - few ulp)
        m = rng.integers(0, 9, nov).astype(np.uint64)
        m = np.where(rng.random(nov) < 0.5, m, np.uint64((1 << 52) - 1) - m)
        eia = _bits(one + m) * 0.5
        eia[::3] = 0.5
        return _bits(one + rng.integers(0, 1 << 52, n).astype(np.uint64)), eia
    if name == "exact":       # multiples of the denominators and their neighbours
        eia = np.full(nov, 1.5) * rng.choice([1.0, -1.0, 3.0, 5.0], nov)
        return np.nextafter(3.0 * rng.integers(1, 1 << 20, n), rng.choice([-np.inf, 0.0, np.inf], n)), eia
    if name == "special":
        x = rng.standard_normal(n)
        x[:8] = [np.inf, -np.inf, np.nan, 0.0, -0.0, 5e-324, 1e308, -1e-308]
        eia = rng.standard_normal(nov)
        eia[:6] = [np.inf, 0.0, -0.0, 1e-310, 1e300, np.nan]
        return rng.permutation(x), eia
    raise KeyError(name)


@pytest.mark.parametrize("name", ["random", "edges", "exact", "special"])
def test_denominators(gpulib, name):
    from fricc_gb300 import _lib as L
    o, v = 3, 37
    rng = np.random.default_rng(len(name))
    x, eia = _inputs(name, o, v, rng)
    x = x.reshape(o, o, v, v)
    e2 = eia.reshape(o, v)
    with np.errstate(all="ignore"):
        want = x / (e2[:, None, :, None] + e2[None, :, None, :])
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    t1, t2, e, z1, z2 = dev(rng.standard_normal(o * v)), dev(x), dev(eia), dev(np.zeros(o * v)), dev(np.zeros(x.size))
    g, fov, res = dev(np.zeros((o * v) ** 2)), dev(np.zeros(o * v)), dev(np.zeros(4))
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    L.check(gpulib.fricc_energy_update(p(t1), p(t2), p(e), p(fov), p(g), p(z1), p(z2), o, v, p(t1), p(t2), p(res),
                                       L.cur_stream()))
    got = t2.cpu().numpy()
    nan = np.isnan(want)
    np.testing.assert_array_equal(np.isnan(got), nan)
    np.testing.assert_array_equal(got[~nan].view(np.int64), want[~nan].view(np.int64))
