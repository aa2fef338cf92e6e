"""The argument plans kept per shape: broadcast strides as torch expands them,
views as torch allows them, and einsum's grouping against torch.einsum."""
import itertools

import pytest
import torch

from fricc_gb300 import rccsd_dense as D


def _views():
    x = torch.arange(2.0 * 3 * 4 * 5, dtype=torch.float64).reshape(2, 3, 4, 5)
    for p in itertools.permutations(range(4)):
        yield x.permute(p)
    yield from (x[:, :1], x[0], x[:, ::2], x[1, 2], x[1, 2, 3, 4], x[:, :, None, 0], x[:1].expand(2, 3, 4, 5))


def test_strides_are_those_of_expand():
    for t in _views():
        for to in {tuple(t.shape), (7, *t.shape)[-5:], tuple(6 if n == 1 else n for n in t.shape)}:
            e = t.expand(to)
            want = [0] * (5 - len(to)) + [s if n != 1 or e.shape == t.shape else s for s, n in zip(e.stride(), to)]
            got = D._strides5(t.shape, t.stride(), to)
            # (the stride of an extent of one is never used)
            dims = [1] * (5 - len(to)) + list(to)
            assert [g for g, n in zip(got, dims) if n > 1] == [w for w, n in zip(want, dims) if n > 1]
    with pytest.raises(RuntimeError):
        D._strides5((2, 3), (3, 1), (2, 4))


def test_viewable_is_torchs_view():
    for t in _views():
        n = t.numel()
        for to in ((1, 1, n), (n, 1, 1), (2, 3, n // 6) if n % 6 == 0 else (1, n, 1), (4, n // 4, 1) if n % 4 == 0 else (n, 1, 1)):
            try:
                t.view(to)
                ok = True
            except RuntimeError:
                ok = False
            assert D._viewable(t.shape, t.stride(), to) == ok
            assert torch.equal(D._as3(t, to), t.reshape(to))


@pytest.mark.parametrize("spec", ["lcki,klac->ia", "kibc,jc->kibj", "ka,kibj->ijab", "lckd,id->lkci", "abc,cd->bd",
                                  "ab,cb->ac", "kij,kja->kia", "ab,bcd->ac", "a,b->ab"])
def test_einsum_plan(spec):
    g = torch.Generator().manual_seed(len(spec))
    size = dict(zip("abcdijkl", (2, 3, 4, 5, 3, 2, 4, 5)))
    a, b = spec.split("->")[0].split(",")
    A, B = (torch.randint(-8, 9, [size[c] for c in t], generator=g).double() for t in (a, b))
    want = torch.einsum(spec, A, B)   # small integers: exact in any order
    assert torch.equal(D.einsum_df(spec, A, B, gemm=D.gemm_torch), want)
    out = want.clone()
    assert torch.equal(D.einsum_df(spec, A, B, gemm=D.gemm_torch, out=out, alpha=2.0, beta=1.0), 3 * want)
