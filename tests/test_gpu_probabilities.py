"""Inclusion probabilities (|x| / R) m' where the quotient is exact, next to a
halfway case, at the ends of the exponent range, or over norms next to a power
of two: values and indices bit for bit the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _x(name):
    rng = np.random.default_rng(len(name))
    if name == "norm_power_of_two":
        x = rng.integers(1, 64, 20_000).astype(float)
        return np.append(x, 2.0 ** 22 - x.sum())
    if name == "norm_above_power":      # the whole norm one unit above 2^20
        x = rng.integers(1, 32, 20_000).astype(float)
        return np.concatenate([[2.0 ** 20 - x.sum()], x, [2.0 ** -32]])
    if name == "small_quotients":       # a / R = k / 3 2^j: the bits repeat
        return 3.0 * rng.integers(1, 9, 24_576) / 2.0 ** rng.integers(0, 30, 24_576)
    if name == "halfway":               # (2^52 + odd) / 2^k over R = 2^k': ties once R is a power of two times 3
        return 1.5 * (1.0 + rng.integers(0, 64, 16_384) * 2.0 ** -52)
    if name == "wide":                  # quotients down to the subnormals
        return rng.random(20_000) * 2.0 ** rng.uniform(-1060, 20, 20_000)
    if name == "subnormal_norm":
        return rng.integers(0, 200, 20_000) * 5e-324
    if name == "random":
        return rng.standard_normal(30_001)
    raise KeyError(name)


@pytest.mark.parametrize("name", ["norm_power_of_two", "norm_above_power", "small_quotients", "halfway", "wide",
                                  "subnormal_norm", "random"])
def test_probabilities_vs_oracle(gpulib, oracle, name):
    from fricc_gb300 import py_rccsd
    x = np.ascontiguousarray(_x(name)).reshape(1, 1, 1, -1)
    m = 3000
    with np.errstate(all="ignore"):
        ref = oracle.SparseTensor4d(x, x.shape, m, "fri", "systematic", rn=0.37)
    flat, vals = py_rccsd.SparseTensor4d(x, x.shape, m, "fri", "systematic", rn=0.37).export()
    np.testing.assert_array_equal(flat, ref.flat)
    np.testing.assert_array_equal(vals.view(np.int64), ref.vals.view(np.int64))
