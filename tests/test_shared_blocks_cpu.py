"""Converted blocks that several solver threads share: none can be seen before
the work that makes it is done, and none is left to be made in the middle of a
solve (CPU: the conversions and streams are stand-ins)."""
import threading
import types

import pytest
import torch

from fricc_gb300 import cholesky
from fricc_gb300 import rccsd_dense as D


class _Stream:
    """A stream whose work completes when the test says so."""

    def __init__(self):
        self.waiting, self.go, self.done = threading.Event(), threading.Event(), False

    def synchronize(self):
        self.waiting.set()
        assert self.go.wait(10)
        self.done = True


@pytest.fixture
def shared(monkeypatch):
    E = D.DeviceERIs.__new__(D.DeviceERIs)
    E.nocc, E.mo_energy = 2, torch.zeros(5)
    E.blk = torch.zeros(9, 4, dtype=torch.float64)
    E._splits, E._mod_bytes, E._lock = {}, 0, threading.Lock()
    st = _Stream()
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: st)
    for mod, name in ((D, "split_f2"), (D, "mod_operand"), (D, "to_f32_rows"), (cholesky, "split_a"),
                      (cholesky, "split_b")):
        monkeypatch.setattr(mod, name, lambda *a: "made")
    lib = types.SimpleNamespace(fricc_mod_bytes=lambda rows, k: 32 * rows * k)
    monkeypatch.setattr(D.L, "load", lambda *a: lib)
    monkeypatch.setattr(D.DeviceERIs, "_free_bytes", staticmethod(lambda *a: 1 << 40))
    return E, st


@pytest.mark.parametrize("make", [lambda E: E.prepare_splits(("blk",)), lambda E: E.mod_w("blk", 4),
                                  lambda E: E.tc_w("blk", 4), lambda E: E.prepare_f32({"blk": 4}),
                                  lambda E: E.prepare_tc({"blk": ("A", 9, 4)})],
                         ids=["pairs", "modular", "tensor", "fp32", "dense"])
def test_no_block_is_seen_in_flight(shared, make):
    E, st = shared
    seen = []

    def second():
        make(E)
        seen.append(st.done)
    a = threading.Thread(target=make, args=(E,))
    a.start()
    assert st.waiting.wait(10)
    b = threading.Thread(target=second)
    b.start()
    b.join(0.2)  # it has to wait for the first one's stream
    assert not seen and not E._splits
    st.go.set()
    a.join(10)
    b.join(10)
    assert seen == [True] and len(E._splits) == 1


@pytest.mark.parametrize("budget,pairs", [(0, ("vvvvT",)), (1 << 30, ())])
def test_pair_blocks_count_the_budget(shared, monkeypatch, budget, pairs):
    """A block that runs as a modular product only once converted, and cannot
    be kept converted, is among those to be made before the first iteration."""
    E, st = shared
    st.go.set()
    E.vvvvT = torch.zeros(9, 9, dtype=torch.float64)
    monkeypatch.setattr(E, "MOD_BYTES", budget, raising=False)
    monkeypatch.setattr(D, "takes_mod", lambda dims, m, term, prepared, pairs_: prepared)
    assert E.pair_blocks(10, False, ("vvvvT",)) == pairs
