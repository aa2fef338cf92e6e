"""The memory a served solve is admitted with counts the converted blocks its
sizes choose, not every block that could be converted."""
import pytest

from fricc_gb300 import _lib as L
from fricc_gb300 import rccsd_dense as D
from fricc_gb300.batch import footprint_bytes


def _plain(o, v):
    return 8 * (2 * v**4 + 9 * o * v**3 + 16 * o * o * v * v + 4 * o**4 + 8 * o**3 * v)


@pytest.mark.parametrize("o,v,m,pairs", [(20, 100, 200_000, True), (20, 100, 200_000, False), (14, 61, 60_000, False),
                                         (5, 20, 1000, True),
                                         (30, 150, 2_000_000, True)])
def test_converted_blocks_are_those_the_routes_take(o, v, m, pairs):
    lib = L.load()
    vvvv = D.takes_mod((o, o, v, v), m, (0, 1, 2, 3, v * v), True, pairs)
    # (vv|vv), X/Y and six ovvv-sized or smaller operands at most
    most = lib.fricc_mod_bytes(v * v, v * v) * vvvv + lib.fricc_mod_bytes(2 * o * v, v * v)
    most += sum(lib.fricc_mod_bytes(M if s == "A" else N, K) for M, N, K, s in D.dense_uses(o, v).values())
    most += 4 * lib.fricc_mod_bytes(o * v, o * v) + 104 * (o * v) ** 2
    got = footprint_bytes(o, v, "df64" if pairs else "fp64", m) - _plain(o, v)
    assert 0 < got <= most
    if vvvv:
        assert got >= lib.fricc_mod_bytes(v * v, v * v)


def test_pairs_keep_the_large_block_unconverted_at_o20v100():
    assert not D.takes_mod((20, 20, 100, 100), 200_000, (0, 1, 2, 3, 10_000), True, True)
    assert footprint_bytes(20, 100, "df64", 200_000) < _plain(20, 100) + 32 * 100**4 + 104 * 2000**2 + 2e9


def test_dense_uses_are_the_products_shapes():
    for o, v in ((3, 7), (20, 100)):
        for name, (M, N, K, side) in D.dense_uses(o, v).items():
            size = {"g_klcd": (o * v) ** 2, "g_kldc": (o * v) ** 2}.get(name, o * v**3)
            assert (M * K if side == "A" else K * N) == size
