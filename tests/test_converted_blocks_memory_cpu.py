"""Integral blocks kept converted take no memory a solve needs: a shortage
leaves a block as it is, once and for all (CPU: stand-ins)."""
import threading
import types

import pytest
import torch

from fricc_gb300 import rccsd_dense as D

SIZE = 1 << 28


@pytest.fixture
def eris(monkeypatch):
    E = D.DeviceERIs.__new__(D.DeviceERIs)
    E.blk = torch.zeros(9, 4, dtype=torch.float64)
    E._splits, E._mod_bytes, E._lock = {}, 0, threading.Lock()
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: types.SimpleNamespace(synchronize=lambda: None))
    monkeypatch.setattr(D.L, "load", lambda *a: types.SimpleNamespace(fricc_mod_bytes=lambda rows, k: SIZE))
    E.made = []
    monkeypatch.setattr(D, "mod_operand", lambda x, *a: E.made.append(a) or "made")
    monkeypatch.setattr(D.DeviceERIs, "_free_bytes", staticmethod(lambda *a: 1 << 30), raising=False)
    return E


def test_kept_and_counted(eris):
    assert eris.mod_w("blk", 4) == "made" and eris.mod_w("blk", 4) == "made"
    assert len(eris.made) == 1 and eris._mod_bytes == SIZE


@pytest.mark.parametrize("free,kept", [(2 * SIZE - 1, None), (2 * SIZE, "made")])
def test_as_much_again_stays_free(eris, monkeypatch, free, kept):
    monkeypatch.setattr(D.DeviceERIs, "_free_bytes", staticmethod(lambda *a: free))
    assert eris.mod_w("blk", 4) == kept


def test_a_failed_allocation_is_no_error(eris, monkeypatch):
    tried = []

    def fails(*a):
        tried.append(a)
        raise torch.OutOfMemoryError("out of memory")
    monkeypatch.setattr(D, "mod_operand", fails)
    assert eris.mod_w("blk", 4) is None and eris.mod_w("blk", 4) is None
    assert len(tried) == 1 and eris._mod_bytes == 0
    assert eris.mod_b("blk", 9, 4) is None and len(tried) == 2
