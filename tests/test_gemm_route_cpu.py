"""fricc_gemm_takes_mod answers for the dispatch it predicts: a constant
operand is never converted for a product that then runs elsewhere."""
import pytest
import torch

from fricc_gb300 import _lib as L
from fricc_gb300 import rccsd_dense as D


@pytest.fixture
def lib():
    lib = L.load()
    assert lib.fricc_mod_select(1) == 0  # wherever possible
    yield lib
    assert lib.fricc_mod_select(-1) == 0 and lib.fricc_tune_set(1, -1) == 0


@pytest.mark.parametrize("M,N,takes", [(4, 500, 0), (500, 4, 0), (1, 1, 0), (5, 5, 1)])
def test_few_rows_or_columns_are_not_taken(lib, M, N, takes):
    assert lib.fricc_gemm_takes_mod(1, M, N, 100, 0, 0, 1, 0, 1) == takes


def test_a_tuned_tile_is_not_taken(lib):
    A, B, C = torch.zeros(50, 30), torch.zeros(30, 40), torch.zeros(50, 40)
    E = type("E", (), {"mod_a": lambda *a: "A", "mod_b": lambda *a: "B"})()
    assert D.mod_constants(E, A, B, C, "x", None, True) == ("A", None)
    assert lib.fricc_tune_set(1, 2) == 0
    assert lib.fricc_gemm_takes_mod(1, 50, 40, 30, 0, 0, 1, 0, 1) == 0
    assert D.mod_constants(E, A, B, C, "x", None, True) == (None, None)
    assert lib.fricc_tune_set(1, -1) == 0
    assert D.mod_constants(E, A, B, C, None, "x", True) == (None, "B")
