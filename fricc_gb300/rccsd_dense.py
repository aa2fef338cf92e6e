"""Dense closed-shell CCSD pieces of one FRI-CCSD iteration, on the GPU (FP64).

These are the parts of fricc/friccsd.py:update_amps that the reference
delegates to PySCF (``rintermediates`` cc_Foo, cc_Fvv, cc_Fov, Loo, Lvv and
the dense W intermediates, the CCSD energy) written from the closed-shell
CCSD equations (Hirata et al., J. Chem. Phys. 120, 2581 (2004)), with torch
tensors on the device.  The reference-shaped helpers below (cc_Foo, Loo,
cc_Woooo, ...) are written with torch einsums and serve the uncompressed
variants and the tests; the iteration itself (fricc_gb300.friccsd) runs its
dense algebra on the library's GEMMs (gemm_f64, gemm_df, the tensor-core
GEMM) and its elementwise passes on the library's combine kernel.

Integral blocks, chemists' notation: ovov[i,a,j,b] = (ia|jb),
oovv[i,j,a,b] = (ij|ab), ovvo[i,a,b,j] = (ia|bj), ovoo[i,a,j,k] = (ia|jk),
ovvv[i,a,b,c] = (ia|bc), oooo[i,j,k,l] = (ij|kl); the vvvv block is kept
only as vvvvT[c,d,a,b] = (ac|bd), the layout the O^2V^4 term streams.
"""
from __future__ import annotations

import functools
import math
import threading

import numpy as np
import torch

from . import _lib as L

ein = torch.einsum


class DeviceERIs:
    """Integrals and orbital energies resident in HBM for the whole solve."""

    def __init__(self, fock, mo_energy, nocc, blocks, device="cuda"):
        dev = torch.device(device)
        f64 = torch.float64

        def put(a):
            return (a if isinstance(a, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(a))).to(
                dev, f64).contiguous()

        self.device = dev
        self.nocc = int(nocc)
        self.fock = put(fock)
        self.mo_energy = put(mo_energy)
        for k in ("oooo", "ovoo", "ovov", "oovv", "ovvo", "ovvv"):
            setattr(self, k, put(blocks[k]))
        vvvv = put(blocks["vvvv"]) if "vvvv" in blocks else None
        if "vvvvT" in blocks:
            self.vvvvT = put(blocks["vvvvT"])
        elif vvvv is not None:
            self.vvvvT = vvvv.permute(1, 3, 0, 2).contiguous()  # [c,d,a,b] = (ac|bd)
        else:
            # split precision: (vv|vv) is rebuilt from the factor when needed
            # (fricc_gb300.cholesky); only sum_cd (ac|bd) is kept
            self.vvvvT = None
        del vvvv
        self._S0 = put(blocks["S0"]) if "S0" in blocks else None
        self.vvvv_rebuild = blocks.get("vvvv_rebuild")
        self._derive()

    def _derive(self):
        """Constant layouts and combinations reused every iteration."""
        ovvv, ovov, ovoo = self.ovvv, self.ovov, self.ovoo
        self.g_ovov = 2.0 * ovov - ovov.permute(0, 3, 2, 1)               # 2(kc|ld) - (kd|lc)
        self.g_ovoo = 2.0 * ovoo - ovoo.permute(2, 1, 0, 3)               # [l,c,k,i]: 2(lc|ki) - (kc|li)
        # T1 O^2V^3 terms as one GEMM: G[k,c,d,a] = 2 (kd|ac) - (kc|ad)
        # and as [k,d,c,a]: X[c,a] = sum_kd t1[k,d] G[k,c,d,a] is one GEMV
        # (it serves the t1.t1 T1 term and the ovvv part of Lvv).  (The ovvv-sized
        # layouts go through the library's elementwise pass: at o18v90 the
        # torch expressions took 440 us.)
        o, v = ovvv.shape[0], ovvv.shape[1]
        new = functools.partial(torch.empty, dtype=ovvv.dtype, device=ovvv.device)
        self.G_t1, self.G_t1_kdca = new(o, v, v, v), new(o, v, v, v)
        _linear([self.G_t1, self.G_t1_kdca.permute(0, 2, 1, 3)], [ovvv.permute(0, 3, 1, 2), ovvv.permute(0, 1, 3, 2)],
                [2.0, -1.0])
        # the T1 terms 2 sum_kc (kc|ai) t_kc - sum_kc (ki|ac) t_kc as one GEMV:
        # G1[k,c,i,a] = 2 (kc|ai) - (ki|ac)
        self.G_t1_kcia = (2.0 * self.ovvo.permute(0, 1, 3, 2) - self.oovv.permute(0, 3, 1, 2)).contiguous()
        # the t1 parts of Wvvvv, contracted with the compressed T2 instead of being
        # built densely: W'[c,d,(x,k,a)] = (kd|ac) for x=0 and (kc|ad) for x=1
        self.ovvv_XY = new(v, v, 2, o, v)
        _linear([self.ovvv_XY[:, :, 0]], [ovvv.permute(3, 1, 0, 2)], [1.0])
        _linear([self.ovvv_XY[:, :, 1]], [ovvv.permute(1, 3, 0, 2)], [1.0])
        # sum_cd of the three Wvvvv pieces (for the reference's Wvvvv.t1.t1 term)
        self.S0 = self._S0 if self._S0 is not None else self.vvvvT.sum(dim=(0, 1))  # [a,b] = sum_cd (ac|bd)
        self.U = ovvv.sum(dim=(1, 3))                                     # [k,a] = sum_cd (kd|ac) = sum_cd (kc|ad)
        # W' of the sparse W-intermediate terms, [l,d,k,c]
        self.ovov_0312 = ovov.permute(0, 3, 2, 1).contiguous()            # (lc|kd)
        self.ovov_0313_0113 = (ovov - 0.5 * ovov.permute(0, 3, 2, 1)).contiguous()
        self.ovov_cdkl = ovov.permute(1, 3, 0, 2).contiguous()            # 1323: [c,d,k,l] = (kc|ld)
        # GEMM-ready layouts for the dense O^2V^3 contractions
        self.g_klcd = self.g_ovov.permute(0, 2, 1, 3).contiguous()       # cc_Foo
        self.g_kldc = self.g_ovov.permute(0, 2, 3, 1).contiguous()       # cc_Fvv
        self.ovvv_iabc, self.ovvv_kacd = new(o, v, v, v), new(o, v, v, v)
        _linear([self.ovvv_iabc], [ovvv.permute(0, 1, 3, 2)], [1.0])      # T2 driver term
        _linear([self.ovvv_kacd], [ovvv.permute(0, 2, 3, 1)], [1.0])      # Wvovo t1 term
        self._dense_wvvvv = None
        self._splits = {}
        self._mod_bytes = 0
        self._lock = threading.Lock()

    SPLIT_BLOCKS = ("vvvvT", "ovvv_XY", "ovov", "ovov_0312", "ovov_0313_0113", "ovov_cdkl")

    def _kept(self, key, make):
        """The form of a constant block kept under ``key``, made once under a
        lock and waited for before it can be seen: solvers on other threads and
        streams never read one whose conversion is still in flight.  (``make``
        may return None: nothing is kept.)"""
        got = self._splits.get(key)
        if got is None:
            with self._lock:
                got = self._splits.get(key)
                if got is None:
                    got = make()
                    if got is not None:
                        torch.cuda.current_stream().synchronize()
                        self._splits[key] = got
        return got

    def prepare_splits(self, names=None):
        """Build the (hi, lo) float-pair forms of constant W' blocks once (by
        default those of FRI-CCSD)."""
        for name in self.SPLIT_BLOCKS if names is None else names:
            if getattr(self, name) is not None:
                self._kept(name, lambda: split_f2(getattr(self, name)))

    def pair_blocks(self, m, every, names=None):
        """The constant W' blocks a df64 solver keeping m entries contracts in
        float pairs: all of them with ``every`` (an autotuner compares the
        float-pair launches), else those whose term does not run as a modular
        tensor-core product (one that does only with the block converted counts
        where that is kept, which is settled here, before the first iteration)."""
        names = self.SPLIT_BLOCKS if names is None else names
        if every:
            return names
        o, v = self.nocc, self.mo_energy.numel() - self.nocc
        use = sparse_uses(o, v)
        dims = (o, o, v, v)

        def modular(n, t):
            return takes_mod(dims, m, t, False, True) or (takes_mod(dims, m, t, True, True) and
                                                          self.mod_w(n, t[4]) is not None)
        return tuple(n for n in names
                     if getattr(self, n) is not None and not all(modular(n, t) for t in use[n]))

    LIN_BLOCKS = ("oooo_klij", "lin_WA", "lin_WB", "lin_W2AB")

    def prepare_linear(self):
        """The bare-integral W' layouts FRI-LCCSD contracts the compressed T2
        with (fricc/frilccsd.py:172-175), built once and shared by solvers:
        oooo_klij[k,l,i,j] = (ki|lj) (0101), lin_WA[k,c,i,a] = (kc|ai)
        (1302, 1303), lin_WB[k,c,i,a] = (ki|ac) (1202, 1203) and
        2 lin_WA - lin_WB (1302 and 1202 from one compression)."""
        if not hasattr(self, "lin_WA"):
            self.oooo_klij = self.oooo.permute(0, 2, 1, 3).contiguous()
            self.lin_WA = self.ovvo.permute(0, 1, 3, 2).contiguous()
            self.lin_WB = self.oovv.permute(0, 3, 1, 2).contiguous()
            self.lin_W2AB = (2.0 * self.lin_WA - self.lin_WB).contiguous()
            if self.device.type == "cuda":
                torch.cuda.current_stream().synchronize()

    def prepare_f32(self, blocks: dict):
        """Build the FP32 forms {name: qs} once."""
        for n, q in blocks.items():
            self.f32(n, q)

    def prepare_tc(self, operands: dict):
        """The split-BF16x3 operands of constant blocks for the split-precision
        form's tensor-core GEMMs, made once:
        {name: ("A" or "B", rows, cols)} with the block viewed as [rows, cols]."""
        from .cholesky import split_a, split_b
        for n, (role, r, c) in operands.items():
            self._kept(("tc", n), lambda: (role, (split_a if role == "A" else split_b)(getattr(self, n).reshape(r, c))))

    def tc_w(self, name, qs):
        """The split W^T ([hi|lo|hi], rows q) of a constant W' block viewed as
        [rows][qs]: the B operand of the split-precision dense sparse terms,
        built on first use (the first, eager iteration)."""
        from .cholesky import split_b
        return self._kept(("tcW", name, qs), lambda: split_b(getattr(self, name).reshape(-1, qs)))

    def tc(self, name, role):
        got = self._splits.get(("tc", name))
        if got is None or got[0] != role:
            raise RuntimeError(f"split operand {role} of {name} missing: call prepare_tc() first")
        return got[1]

    # device bytes of integral blocks kept converted for the modular products, at
    # most (a seventh of the card; four times the FP64 blocks': all of them at
    # o30v150 take 39 GB); a block beyond that is converted by each call that
    # uses it
    MOD_BYTES = 40 << 30

    @staticmethod
    def _free_bytes(enough):
        """Device memory this process could still take: free, and (asked for,
        ~150 us, only where that is not ``enough``) cached unused."""
        free, _ = torch.cuda.mem_get_info()
        return free if free >= enough else free + torch.cuda.memory_reserved() - torch.cuda.memory_allocated()

    def _mod(self, key, name, rows, k, row_stride, k_stride):
        got = self._splits.get(key)
        if got is not None:
            return got
        # settled once per block: beyond the budget, or where as much again would
        # not stay free (a solve that fits without it has to go on fitting), it is
        # not kept
        if ("not", key) in self._splits:
            return None

        def make():
            need = L.load().fricc_mod_bytes(rows, k)
            # (a thousandth of the card is not worth the question)
            roomy = need < 1 << 28 or 2 * need <= self._free_bytes(2 * need)
            if self._mod_bytes + need <= self.MOD_BYTES and roomy:
                try:
                    got = mod_operand(getattr(self, name), rows, k, row_stride, k_stride)
                    self._mod_bytes += need
                    return got
                except torch.OutOfMemoryError:
                    pass
            self._splits[("not", key)] = True
            return None
        return self._kept(key, make)

    def mod_w(self, name, qs):
        """A constant W' block viewed as [keys][qs], its rows q prepared for
        the modular products, built on first use (None where it is not kept)."""
        return self._mod(("modW", name, qs), name, qs, getattr(self, name).numel() // qs, 1, qs)

    def mod_a(self, name, m, k):
        """A constant block as the A operand [m, k] of a dense product."""
        return self._mod(("modA", name, m, k), name, m, k, k, 1)

    def mod_b(self, name, k, n):
        """A constant block as the B operand [k, n] of a dense product."""
        return self._mod(("modB", name, k, n), name, n, k, 1, n)

    def f32(self, name, qs):
        """FP32 rows (qs columns, padded to even) of a constant block, built
        once: the W' operands of the split-precision form."""
        return self._kept(("f32", name, qs), lambda: to_f32_rows(getattr(self, name), qs))

    def split(self, name):
        """The float-pair form of a constant block (prepare_splits() built it)."""
        if name not in self._splits:
            raise RuntimeError(f"float-pair form of {name} missing: call prepare_splits() first")
        return self._splits[name]

    @property
    def ovvv_kcda(self):  # [k,c,d,a] = (kd|ac), only for the dense Wvvvv build
        return self.ovvv.permute(0, 3, 1, 2).contiguous()

    @property
    def ovvv_cdkb(self):  # [c,d,k,b] = (kc|bd), only for the dense Wvvvv build
        return self.ovvv.permute(1, 3, 0, 2).contiguous()

    @classmethod
    def from_system(cls, system, device="cuda"):
        """Build every block on the device from the Cholesky factor of a SyntheticSystem."""
        dev = torch.device(device)
        L = _dev_tensor(system.L, dev)
        o = system.nocc
        naux = L.shape[0]
        sl = {"o": slice(0, o), "v": slice(o, system.nmo)}

        def blk(name):
            p, q, r, s = (sl[c] for c in name)
            A = L[:, p, q].reshape(naux, -1)
            B = L[:, r, s].reshape(naux, -1)
            n1 = L[:, p, q].shape[1:]
            n2 = L[:, r, s].shape[1:]
            return (A.T @ B).reshape(*n1, *n2)

        blocks = {k: blk(k) for k in ("oooo", "ovoo", "ovov", "oovv", "ovvv")}
        # (ia|bj) = (ia|jb): L is symmetric in its two orbital indices
        blocks["ovvo"] = blocks["ovov"].permute(0, 1, 3, 2).contiguous()
        Lvv = L[:, sl["v"], sl["v"]]
        v = system.nvir
        # vvvvT[c,d,a,b] = (ac|bd) = sum_P L[P,a,c] L[P,b,d]
        Lca = Lvv.permute(0, 2, 1).reshape(naux, v * v)  # [P, (c,a)]
        Ldb = Lvv.permute(0, 2, 1).reshape(naux, v * v)  # [P, (d,b)]
        X = (Lca.T @ Ldb).reshape(v, v, v, v)            # [c,a,d,b]
        blocks["vvvvT"] = X.permute(0, 2, 1, 3).contiguous()
        del X
        return cls(_dev_tensor(system.fock, dev), _dev_tensor(system.mo_energy, dev), o, blocks, device)

    def to_numpy_blocks(self):
        """Host copies in the stand-in layout (for checking against the oracle)."""
        out = {k: getattr(self, k).cpu().numpy() for k in ("oooo", "ovoo", "ovov", "oovv", "ovvo", "ovvv")}
        out["vvvv"] = self.vvvvT.permute(2, 0, 3, 1).contiguous().cpu().numpy()  # (ab|cd)
        return out


def sym_add(out: torch.Tensor, X: torch.Tensor, coef: float = 1.0) -> torch.Tensor:
    """out += coef * (X + X.permute(1, 0, 3, 2)) in one fused pass (the
    symmetrised T2 residual terms); out contiguous [o,o,v,v] FP64 on the
    device, X any [o,o,v,v] FP64 view not overlapping out."""
    import ctypes

    o, v = out.shape[0], out.shape[2]
    if (not out.is_contiguous() or out.dtype != torch.float64 or X.dtype != torch.float64
            or tuple(X.shape) != tuple(out.shape) or out.shape != (o, o, v, v)):
        raise ValueError("sym_add: out contiguous [o,o,v,v] float64 and X a float64 view of the same shape")
    L.check(L.load().fricc_symadd(ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(X.data_ptr()), o, v,
                                  L.i64arr(X.stride()), float(coef),
                                  L.cur_stream()))
    return out


def _sig(ts):
    return tuple((t.shape, t.stride()) for t in ts)


def _strides5(shape, stride, to):
    """Element strides of a (shape, stride) tensor broadcast to ``to``, padded
    to 5 dims."""
    n = len(to) - len(shape)
    if n < 0 or any(a != b and a != 1 for a, b in zip(shape, to[n:])):
        raise RuntimeError(f"combine: cannot broadcast {tuple(shape)} to {tuple(to)}")
    return [0] * (5 - len(shape)) + [s if a == b else 0 for s, a, b in zip(stride, shape, to[n:])]


# What the argument arrays of one combine call hold besides the pointers
# depends on shapes and strides alone: an iteration makes ~45 such calls and
# building them took ~15 of the ~25 us of each (o10v40 is bound by the host).
# The library only reads the arrays, so threads share them.
@functools.lru_cache(maxsize=4096)
def _combine_plan(outs, xs, prod):
    shape = tuple(outs[0][0])
    if len(shape) > 5 or any(tuple(o[0]) != shape for o in outs):
        raise ValueError("combine: outputs of one shape, at most 5 dims")
    dims = [1] * (5 - len(shape)) + list(shape)
    # walk the index space in the first output's memory order (its
    # smallest stride innermost), so its reads and writes coalesce
    s0 = _strides5(*outs[0], shape)
    perm = sorted(range(5), key=lambda d: (dims[d] != 1, -s0[d]))

    def strides(sig):
        flat = []
        for sh, st in sig:
            s5 = _strides5(sh, st, shape)
            flat.extend(s5[d] for d in perm)
        return L.i64arr(flat if flat else [0])

    return L.i64arr([dims[d] for d in perm]), strides(xs), strides(prod), strides(outs)


def _ptrs(ts):
    import ctypes

    return (ctypes.c_void_p * (len(ts) or 1))(*[t.data_ptr() for t in ts])


def combine(outs, xs=(), coefs=None, prod=(), accumulate=False):
    """One pass of the library's strided elementwise kernel (fricc_combine5):
    out_k = sum_t coefs[k][t] xs[t] (+ coefs[k][-1] * prod[0] * prod[1] ...
    when ``prod`` is given), or out_k += that with ``accumulate``.  Every
    tensor is an FP64 device view; inputs broadcast to the outputs' shape
    (at most 5 dims); the kernel walks the first output's memory order.
    Outputs must not overlap the inputs."""
    import ctypes

    outs, xs, prod = list(outs), list(xs), list(prod)
    for t in outs + xs + prod:
        if t.dtype != torch.float64 or not t.is_cuda:
            raise ValueError("combine: FP64 CUDA tensors only")
    nc = len(xs) + (1 if prod else 0)
    if coefs is None:
        coefs = [[1.0] * nc for _ in outs]
    dims, sx, sp, so = _combine_plan(_sig(outs), _sig(xs), _sig(prod))
    if len(coefs) != len(outs) or any(len(c) != nc for c in coefs):
        raise ValueError("combine: one coefficient per input (and one for the product) per output")
    cf = (ctypes.c_double * (len(outs) * nc))(*[float(c) for row in coefs for c in row])
    L.check(L.load().fricc_combine5(dims, len(xs), _ptrs(xs), sx, len(prod), _ptrs(prod), sp, len(outs), _ptrs(outs), so,
                                    cf, int(bool(accumulate)), L.cur_stream()))
    return outs[0]


def _linear(outs, xs, coefs):
    """Every out = sum_t coefs[t] xs[t]: one combine on the device, torch on a
    host tensor."""
    if outs[0].is_cuda:
        combine(outs, xs, [list(coefs) for _ in outs])
        return
    r = sum(c * x for c, x in zip(coefs, xs))
    for out in outs:
        out.copy_(r)


def zero(t: torch.Tensor) -> torch.Tensor:
    """t[...] = 0 for a contiguous device tensor, through the library."""
    import ctypes

    if not t.is_contiguous():
        raise ValueError("zero: contiguous tensors only")
    L.check(L.load().fricc_zero(ctypes.c_void_p(t.data_ptr()), t.numel() * t.element_size(),
                                L.cur_stream()))
    return t


def _dev_tensor(a, dev):
    """FP64 copy of a numpy array, or the tensor itself moved to ``dev``."""
    t = a if isinstance(a, torch.Tensor) else torch.from_numpy(np.ascontiguousarray(a))
    return t.to(dev, torch.float64)


def _strides3(t: torch.Tensor):
    if t.dim() == 2:
        return (t.stride(0), t.stride(1), 0), 1
    return (t.stride(1), t.stride(2), t.stride(0)), t.shape[0]


def _bstrides(shape, stride):
    """(row, col, batch, batch2) element strides and (batch, batch2) extents of
    a 2-D, 3-D ([batch, M, K]) or 4-D ([batch2, batch, M, K]) operand."""
    if len(shape) == 2:
        return (stride[0], stride[1], 0, 0), 1, 1
    if len(shape) == 3:
        return (stride[1], stride[2], stride[0], 0), shape[0], 1
    if len(shape) == 4:
        return (stride[2], stride[3], stride[1], stride[0]), shape[1], shape[0]
    raise ValueError("gemm: operands are 2-D, 3-D or 4-D")


@functools.lru_cache(maxsize=4096)
def _gemm_plan(A, B, C):
    """(batch, batch2, M, N, K, stride arrays of three, of four) of operands
    given as (shape, stride); the library only reads the arrays."""
    sA, bA, b2A = _bstrides(*A)
    sB, bB, b2B = _bstrides(*B)
    sC, batch, batch2 = _bstrides(*C)
    M, N = C[0][-2], C[0][-1]
    K = A[0][-1]
    assert A[0][-2] == M and B[0][-2] == K and B[0][-1] == N
    assert bA in (1, batch) and bB in (1, batch) and b2A in (1, batch2) and b2B in (1, batch2)
    # a size-1 batch level of an operand is shared: stride 0
    sA = (sA[0], sA[1], sA[2] if bA == batch and batch > 1 else 0, sA[3] if b2A == batch2 and batch2 > 1 else 0)
    sB = (sB[0], sB[1], sB[2] if bB == batch and batch > 1 else 0, sB[3] if b2B == batch2 and batch2 > 1 else 0)
    return (batch, batch2, M, N, K, tuple(L.i64arr(x[:3]) for x in (sA, sB, sC)),
            tuple(L.i64arr(x) for x in (sA, sB, sC)))


def _gemm_call(fn, A, B, C, alpha, beta):
    batch, batch2, M, N, K, s3, s4 = _gemm_plan(*_sig((A, B, C)))
    lib = L.load()
    if batch2 == 1:
        L.check(getattr(lib, fn)(A.data_ptr(), B.data_ptr(), C.data_ptr(), batch, M, N, K, *s3, float(alpha), float(beta),
                                 L.cur_stream()))
    else:
        L.check(getattr(lib, fn + "_b2")(A.data_ptr(), B.data_ptr(), C.data_ptr(), batch, batch2, M, N, K, *s4,
                                         float(alpha), float(beta), L.cur_stream()))
    return C


def gemm_df(A: torch.Tensor, B: torch.Tensor, C: torch.Tensor, alpha: float = 1.0, beta: float = 0.0):
    """C = alpha A @ B + beta C on the FP32-pair GEMM kernel; FP64 tensors with
    any strides, 2-D or batched 3-D (a batch stride of 0 shares an operand)."""
    return _gemm_call("fricc_gemm_df", A, B, C, alpha, beta)


def gemm_f64(A: torch.Tensor, B: torch.Tensor, C: torch.Tensor, alpha: float = 1.0, beta: float = 0.0,
             a_mod=None, b_mod=None):
    """The same contract in FP64: the library's DFMA kernel, or, for large
    products, its modular tensor-core product at the same accuracy.
    ``a_mod`` / ``b_mod``: a 2-D operand prepared once (``mod_operand``)."""
    if a_mod is None and b_mod is None:
        return _gemm_call("fricc_gemm_f64", A, B, C, alpha, beta)
    batch, batch2, M, N, K, _, s4 = _gemm_plan(*_sig((A, B, C)))
    L.check(L.load().fricc_gemm_f64_mod(
        A.data_ptr(), a_mod.data_ptr() if a_mod is not None else None, B.data_ptr(),
        b_mod.data_ptr() if b_mod is not None else None, C.data_ptr(), batch, batch2, M, N, K, *s4, float(alpha),
        float(beta), L.cur_stream()))
    return C


def sparse_uses(o, v):
    """The sparse terms (pa, pb, ka, kb, QS) each constant W' block serves."""
    ov = o * v
    return {"vvvvT": [(0, 1, 2, 3, v * v)], "ovvv_XY": [(0, 1, 2, 3, 2 * ov)], "ovov": [(3, 0, 1, 2, ov)],
            "ovov_0312": [(3, 0, 1, 2, ov)], "ovov_0313_0113": [(2, 0, 1, 3, ov)], "ovov_cdkl": [(0, 1, 2, 3, o * o)],
            "oooo_klij": [(2, 3, 0, 1, o * o)], "lin_WA": [(1, 3, 0, 2, ov), (1, 2, 0, 3, ov)],
            "lin_WB": [(1, 3, 0, 2, ov), (1, 2, 0, 3, ov)], "lin_W2AB": [(1, 3, 0, 2, ov)]}


def dense_uses(o, v):
    """The dense products (M, N, K) of FRI-CCSD with a constant block, and
    which operand it is."""
    return {"g_klcd": (o, o, o * v * v, "A"), "g_kldc": (v, v, o * o * v, "B"), "G_t1": (o, v, o * v * v, "B"),
            "ovvv_iabc": (o * v * v, o, v, "A"), "ovvv": (o * v * v, o, v, "A"), "ovvv_kacd": (o * v * v, o, v, "A")}


def converted_bytes(o, v, m, pairs) -> int:
    """Device bytes a FRI-CCSD solve keeping m entries takes for the modular
    products: the constant blocks its sizes let it keep converted
    (DeviceERIs.MOD_BYTES at most), and the scratch of one product (planes and
    residues of amplitude-sized operands).  0 where no term runs so."""
    lib = L.load()
    uses = sparse_uses(o, v)
    kept, dims = 0, (o, o, v, v)
    for name in DeviceERIs.SPLIT_BLOCKS:
        pa, pb, ka, kb, qs = uses[name][0]
        if takes_mod(dims, m, uses[name][0], True, pairs):
            kept += lib.fricc_mod_bytes(qs, dims[ka] * dims[kb])
    for M, N, K, side in dense_uses(o, v).values():
        if gemm_takes_mod(M, N, K, side == "A", side == "B", pairs):
            kept += lib.fricc_mod_bytes(M if side == "A" else N, K)
    return min(kept, DeviceERIs.MOD_BYTES) + (104 * (o * v) ** 2 if kept else 0)


def takes_mod(dims, m, term, prepared, pairs) -> bool:
    """Whether the sparse term (pa, pb, ka, kb, QS) of a T with m entries runs
    as a modular tensor-core product (fricc_spmm_takes_mod)."""
    return _spmm_route(tuple(dims), int(m), term, bool(prepared), bool(pairs), L.load().fricc_mod_mode())


GEMM_TILE = 1  # fricc_tune_set's knob


# (the routes are pure functions of the sizes, the thread's fricc_mod_select mode
# and, for GEMMs, its tile knob; an iteration asks ~30 times, ~3 us each through
# ctypes)
@functools.lru_cache(maxsize=4096)
def _spmm_route(dims, m, term, prepared, pairs, mode):
    pa, pb, ka, kb, qs = term
    return bool(L.load().fricc_spmm_takes_mod(L.i64arr(dims), m, pa, pb, ka, kb, qs, int(prepared), int(pairs)))


@functools.lru_cache(maxsize=4096)
def _gemm_route(M, N, K, a_prepared, b_prepared, pairs, mode, tile):
    return bool(L.load().fricc_gemm_takes_mod(1, M, N, K, 0, 0, int(a_prepared), int(b_prepared), int(pairs)))


def gemm_takes_mod(M, N, K, a_prepared, b_prepared, pairs) -> bool:
    """Whether a dense product of this shape runs as a modular one
    (fricc_gemm_takes_mod)."""
    lib = L.load()
    return _gemm_route(M, N, K, bool(a_prepared), bool(b_prepared), bool(pairs), lib.fricc_mod_mode(),
                       lib.fricc_tune_value(GEMM_TILE))


def mod_constants(E, A, B, C, const, const_b, pairs):
    """The prepared forms (A, B) of the constant integral operands of a dense
    product A @ B (named const / const_b), where it runs as a modular one
    with them; (None, None) elsewhere."""
    if const is None and const_b is None:
        return None, None
    M, N, K = C.shape[-2], C.shape[-1], A.shape[-1]
    if not gemm_takes_mod(M, N, K, const is not None, const_b is not None, pairs):
        return None, None
    return (E.mod_a(const, M, K) if const else None), (E.mod_b(const_b, K, N) if const_b else None)


def mod_operand(x: torch.Tensor, rows: int, k: int, row_stride: int, k_stride: int) -> torch.Tensor:
    """rows x k elements of x converted once for the modular tensor-core
    products (fricc_mod_prepare), as a byte buffer."""
    import ctypes

    lib = L.load()
    buf = torch.empty(lib.fricc_mod_bytes(rows, k), dtype=torch.uint8, device=x.device)
    L.check(lib.fricc_mod_prepare(ctypes.c_void_p(x.data_ptr()), rows, k, row_stride, k_stride,
                                  ctypes.c_void_p(buf.data_ptr()), L.cur_stream()))
    return buf


def _as3(x: torch.Tensor, shape3):
    """x (a permuted view) as a [batch, rows, cols] view, copied to a
    contiguous buffer by the library when its strides do not allow one."""
    if _viewable(x.shape, x.stride(), shape3):
        return x.view(shape3)
    if not x.is_cuda:
        return x.reshape(shape3)
    buf = torch.empty(x.shape, dtype=x.dtype, device=x.device)
    combine([buf], [x])
    return buf.view(shape3)


@functools.lru_cache(maxsize=4096)
def _viewable(shape, stride, to) -> bool:
    try:
        torch.empty_strided(shape, stride, device="meta").view(to)
    except RuntimeError:
        return False
    return True


@functools.lru_cache(maxsize=1024)
def _einsum_plan(spec, shape_a, shape_b):
    lhs, outs = spec.replace(" ", "").split("->")
    a, b = lhs.split(",")
    if len(set(a)) != len(a) or len(set(b)) != len(b):
        raise ValueError(f"einsum_df: repeated index within an operand in {spec!r}")
    size = {c: shape_a[a.index(c)] for c in a}
    size.update({c: shape_b[b.index(c)] for c in b})
    lone_a = [a.index(c) for c in a if c not in b and c not in outs]
    lone_b = [b.index(c) for c in b if c not in a and c not in outs]
    a = "".join(c for c in a if c in b or c in outs)
    b = "".join(c for c in b if c in a or c in outs)
    bt = [c for c in outs if c in a and c in b]
    mi = [c for c in outs if c in a and c not in b]
    ni = [c for c in outs if c in b and c not in a]
    ki = [c for c in a if c in b and c not in outs]
    nb, M, N, K = (math.prod(size[c] for c in idx) for idx in (bt, mi, ni, ki))
    order = bt + mi + ni
    return (lone_a, lone_b, [a.index(c) for c in bt + mi + ki], [b.index(c) for c in bt + ki + ni], (nb, M, K), (nb, K, N),
            (nb, M, N), [size[c] for c in order], [outs.index(c) for c in order], [order.index(c) for c in outs])


def einsum_df(spec: str, A: torch.Tensor, B: torch.Tensor, gemm=None, out=None, alpha: float = 1.0,
              beta: float = 0.0) -> torch.Tensor:
    """Two-operand einsum as one strided batched GEMM on the FP32-pair kernel.

    Indices shared by both operands and the output form the batch, A-only
    output indices the rows, B-only output indices the columns, shared
    non-output indices the contraction; an index in one operand only and not
    in the output is summed out first.  ``gemm`` replaces the FP32-pair GEMM
    (the FP64 form passes the DFMA one, the split-precision form the
    tensor-core one).  Operand groups merge into one stride where the layout
    allows (the library copies them otherwise).  Without ``out`` the result
    is a view of a new contiguous [batch, rows, cols] buffer in the output's
    order; with ``out`` (a tensor in the output's index order whose
    [batch, rows, cols] grouping is a view) the GEMM writes
    out = alpha * result + beta * out in place."""
    lone_a, lone_b, pa, pb, sa, sb, sc, size_c, pc, po = _einsum_plan(spec, A.shape, B.shape)
    if lone_a:
        A = A.sum(dim=lone_a)
    if lone_b:
        B = B.sum(dim=lone_b)
    Ap, Bp = _as3(A.permute(pa), sa), _as3(B.permute(pb), sb)
    K = sa[2]
    if out is not None:
        C = out.permute(pc).view(sc)
    else:
        C = torch.empty(sc, dtype=torch.float64, device=A.device)
        alpha, beta = 1.0, 0.0
    if C.numel():
        if K == 0:
            if beta == 0.0:
                C.zero_()
        else:
            (gemm or gemm_df)(Ap, Bp, C, alpha, beta)
    if out is not None:
        return out
    return C.view(size_c).permute(po)


def gemm_torch(A, B, C, alpha=1.0, beta=0.0):
    """The same contract on cuBLAS FP64."""
    R = torch.matmul(A, B)
    if beta == 0.0:
        C.copy_(R.mul_(alpha) if alpha != 1.0 else R)
    else:
        if beta != 1.0:
            C.mul_(beta)
        C.add_(R, alpha=alpha)
    return C


def to_f32_rows(x: torch.Tensor, qs: int) -> torch.Tensor:
    """x viewed as [rows][qs] in FP32, rows padded to an even length (the
    layout fricc_spmm_f1 reads as float pairs)."""
    rows = x.numel() // qs
    x2 = x.reshape(rows, qs)
    if qs % 2 == 0:
        return x2.to(torch.float32).contiguous()
    out = torch.zeros(rows, qs + 1, dtype=torch.float32, device=x.device)
    out[:, :qs] = x2
    return out


def split_f2(x: torch.Tensor, qs: int = None) -> torch.Tensor:
    """W' [rows][qs] (FP64) as float pairs hi + lo = x (to 2^-47), in the
    q-pair layout of fricc_spmm_f2: per row, float4 (hi_q, hi_q+1, lo_q,
    lo_q+1) for q = 0, 2, 4, ...  qs defaults to the product of the
    dimensions after the first two (W' is always [key1, key2, q...])."""
    import ctypes

    x = x.contiguous()
    if qs is None:
        qs = math.prod(x.shape[2:]) if x.dim() > 2 else x.shape[-1]
    rows = x.numel() // qs
    out = torch.empty(rows * ((qs + 1) // 2) * 4, dtype=torch.float32, device=x.device)
    L.check(L.load().fricc_split_f2(ctypes.c_void_p(x.data_ptr()), rows, qs, ctypes.c_void_p(out.data_ptr()),
                                    L.cur_stream()))
    return out


def cc_Foo(t1, t2, E):
    o = t1.shape[0]
    tt = t2 + ein("ic,ld->ilcd", t1, t1)
    return E.fock[:o, :o] + ein("kcld,ilcd->ki", E.g_ovov, tt)


def cc_Fvv(t1, t2, E):
    o = t1.shape[0]
    tt = t2 + ein("ka,ld->klad", t1, t1)
    return E.fock[o:, o:] - ein("kcld,klad->ac", E.g_ovov, tt)


def cc_Fov(t1, t2, E):
    o = t1.shape[0]
    return E.fock[:o, o:] + ein("kcld,ld->kc", E.g_ovov, t1)


def Loo(t1, t2, E, Foo=None):
    o = t1.shape[0]
    fov = E.fock[:o, o:]
    F = cc_Foo(t1, t2, E) if Foo is None else Foo
    return F + fov @ t1.T + ein("lcki,lc->ki", E.g_ovoo, t1)


def Lvv(t1, t2, E, Fvv=None):
    o = t1.shape[0]
    fov = E.fock[:o, o:]
    F = cc_Fvv(t1, t2, E) if Fvv is None else Fvv
    return F - t1.T @ fov + 2.0 * ein("kdac,kd->ac", E.ovvv, t1) - ein("kcad,kd->ac", E.ovvv, t1)


def cc_Woooo(t1, t2, E):
    W = ein("lcki,jc->klij", E.ovoo, t1)
    W = W + ein("kclj,ic->klij", E.ovoo, t1)
    W = W + ein("kcld,ijcd->klij", E.ovov, t2 + ein("ic,jd->ijcd", t1, t1))
    return W + E.oooo.permute(0, 2, 1, 3)


def cc_Wvoov(t1, t2, E):
    W = ein("kcad,id->akic", E.ovvv, t1)
    W = W - ein("kcli,la->akic", E.ovoo, t1)
    W = W + E.ovvo.permute(2, 0, 3, 1)
    W = W - 0.5 * ein("ldkc,ilda->akic", E.ovov, t2)
    W = W - 0.5 * ein("lckd,ilad->akic", E.ovov, t2)
    W = W + ein("ldkc,ilad->akic", E.ovov, t2)
    return W - ein("ldkc,id,la->akic", E.ovov, t1, t1)


def cc_Wvovo(t1, t2, E):
    W = ein("kdac,id->akci", E.ovvv, t1)
    W = W - ein("lcki,la->akci", E.ovoo, t1)
    W = W + E.oovv.permute(2, 0, 3, 1)
    W = W - 0.5 * ein("lckd,ilda->akci", E.ovov, t2)
    return W - ein("lckd,id,la->akci", E.ovov, t1, t1)


def wvvvv_T(t1, E, out=None):
    """Wvvvv of fricc/friccsd.py:325-331 in the streamed layout [c,d,a,b]:
    (ac|bd) - sum_k (kd|ac) t_kb - sum_k (kc|bd) t_ka."""
    o, v = t1.shape
    W = E.vvvvT.clone() if out is None else out.copy_(E.vvvvT)
    Wf = W.view(v * v, v, v)  # [(c,d), a, b]
    # - sum_k (kd|ac) t_kb  ->  [c,d,a] x [k] . [k,b]
    Wf.view(v * v * v, v).addmm_(E.ovvv_kcda.view(o, v * v * v).T, t1, alpha=-1.0)
    # - sum_k (kc|bd) t_ka  ->  per (c,d): t1^T [a,k] @ (kc|bd)[k,b]
    Wf.baddbmm_(t1.T.unsqueeze(0).expand(v * v, v, o), E.ovvv_cdkb.view(v * v, o, v), alpha=-1.0)
    return W


def wvvvv_sum_cd(t1, E):
    """S[a,b] = sum_cd Wvvvv[a,b,c,d] without building Wvvvv:
    sum_cd (ac|bd) - sum_k t_kb sum_cd (kd|ac) - sum_k t_ka sum_cd (kc|bd)."""
    return E.S0 - E.U.T @ t1 - t1.T @ E.U


def lin_cc_energy(t1, t2, E):
    """2 sum f_ia t1_ia + sum t2_ijab (2 (ia|jb) - (ib|ja)) (fricc/frilccsd.py:504-522)."""
    o = t1.shape[0]
    fov = E.fock[:o, o:]
    return float(2.0 * (fov * t1).sum() + ein("ijab,iajb->", t2, E.g_ovov))


def ccsd_energy(t1, t2, E):
    o = t1.shape[0]
    fov = E.fock[:o, o:]
    tau = t2 + ein("ia,jb->ijab", t1, t1)
    return float(2.0 * (fov * t1).sum() + ein("ijab,iajb->", tau, E.g_ovov))
