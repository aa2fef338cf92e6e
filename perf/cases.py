"""The work a user of this framework has it do, as measurable cases.

Each case is one call (or one loop body) a user's program makes through the
public entry points: the FRI compressions of a T2 tensor, the drop-in
``py_rccsd`` binding, FRI-CCSD and FRI-LCCSD iterations in each arithmetic
form, a replica batch's step, and the integral build of a served request.
Sizes are those of the named workloads and tests of this repository, plus
odd ones of the same ranges.  Systems follow fricc_gb300.synthetic's recipe
(orbital energies uniform, a normalised random Cholesky factor, MP2 T2),
drawn on the GPU; T1 is small and non-zero, as after the first iteration.

``exact`` evaluates the same quantities in plain numpy and torch FP64 from
the reference's definitions, with every sparse term as a dense contraction
with the compressed T2.
"""
from __future__ import annotations

import ctypes
import math
from types import SimpleNamespace

import numpy as np
import torch

from fricc_gb300 import _lib, cholesky, frilccsd, friccsd, py_rccsd, replicas, rccsd_dense, rng

F64 = torch.float64
TERMS = py_rccsd.TERMS


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def _case(kind, o, v, m, naux=None, sigma=0.04, **more):
    return dict(kind=kind, o=o, v=v, m=m, naux=naux or 8 * (o + v), sigma=sigma, **more)


def listed():
    return [
        # one compression of the smallest named workload: latency and launches
        dict(_case("compress", 10, 40, 20_000, 200, 0.05), name="compress_o10v40"),
        # one compression of the headline workload (20 M amplitudes, 10% kept)
        dict(_case("compress", 30, 150, 2_000_000, 900, 0.03), name="compress_o30v150"),
        # the binding's default sampler, at an odd size
        dict(_case("pivotal", 13, 57, 27_000), name="pivotal_o13v57"),
        # the drop-in binding as fricc/friccsd.py drives it: host numpy
        # arrays, one compression and the eleven terms
        dict(_case("binding", 10, 40, 20_000, 200, 0.05, host=True), name="binding_host_o10v40"),
        # the same binding on device tensors at an odd size, 5% kept
        dict(_case("binding", 23, 97, 250_000, host=False), name="binding_dev_o23v97"),
        # one FRI-CCSD iteration with its energy read, as the solver's loop
        # runs it: the smallest named workload (FP64) ...
        dict(_case("iterate", 10, 40, 20_000, 200, 0.05, precision="fp64"), name="iter_fp64_o10v40"),
        # ... the headline workload (FP64) ...
        dict(_case("iterate", 30, 150, 2_000_000, 900, 0.03, precision="fp64"), name="iter_fp64_o30v150"),
        # ... an ordinary size in FP32 pairs ...
        dict(_case("iterate", 20, 100, 200_000, 600, 0.04, precision="df64"), name="iter_df64_o20v100"),
        # ... and the largest workload, split precision
        dict(_case("iterate", 40, 200, 3_200_000, 1200, 0.025, precision="split"), name="iter_split_o40v200"),
        # one step of a fused replica batch (its default arithmetic)
        dict(_case("replicas", 20, 100, 200_000, 600, 0.04, precision="df64", replicas=16),
             name="replicas_df64_o20v100x16"),
        # the integral build in front of a served request
        dict(_case("build", 18, 90, 0), name="build_split_o18v90"),
        # one FRI-LCCSD iteration, odd size
        dict(_case("linear", 14, 61, 60_000, precision="fp64"), name="lccsd_fp64_o14v61"),
    ]


def draw(rng_):
    """A case of the same ranges: nocc from 5 up, nvir = 4 to 6 nocc, 5% to
    20% of T2 kept, naux = 8 (nocc + nvir) (the served stream's recipe)."""
    kind = rng_.choice(["compress", "compress", "pivotal", "binding", "iterate", "iterate", "iterate", "replicas",
                        "build", "linear"])
    precision = rng_.choice(["fp64", "fp64", "df64", "split"]) if kind == "iterate" else \
        rng_.choice(["fp64", "df64"])
    host = rng_.random() < 0.5
    hi = {"compress": 30, "pivotal": 18, "binding": 11 if host else 24, "replicas": 20, "build": 24,
          "linear": 24}.get(kind, {"fp64": 26, "df64": 28, "split": 34}[precision])
    lo = 10 if precision == "split" else 5
    o = int(round(math.exp(rng_.uniform(math.log(lo), math.log(hi)))))
    v = min(int(math.ceil(rng_.uniform(4.0, 6.0) * o)), 5 * hi)
    n = (o * v) ** 2
    m = 0 if kind == "build" else int(n * rng_.uniform(0.05, 0.20))
    more = {}
    if kind == "binding":
        more["host"] = host
    if kind in ("iterate", "linear", "replicas"):
        more["precision"] = precision
    if kind == "replicas":
        more["replicas"] = rng_.randint(2, 8)
    return _case(kind, o, v, m, **more)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _system(case, seed):
    """A synthetic closed-shell system (the attributes DeviceERIs.from_system
    and split_eris read)."""
    o, v, naux = case["o"], case["v"], case["naux"]
    nmo = o + v
    g = _generator(seed)
    eo = torch.sort(torch.rand(o, generator=g, device="cuda", dtype=F64) * 1.2 - 1.5).values
    ev = torch.sort(torch.rand(v, generator=g, device="cuda", dtype=F64) * 2.8 + 0.2).values
    mo = torch.cat([eo, ev])
    A = torch.randn(naux, nmo, nmo, generator=g, device="cuda", dtype=F64) * (case["sigma"] / naux ** 0.5)
    L = torch.triu(A) + torch.triu(A, 1).transpose(1, 2)
    t1 = torch.randn(o, v, generator=g, device="cuda", dtype=F64) * 2e-3
    rn = torch.rand(6, generator=g, device="cuda", dtype=F64).tolist()
    return SimpleNamespace(nocc=o, nvir=v, nmo=nmo, naux=naux, mo_energy=mo, fock=torch.diag(mo), L=L, t1=t1, rn=rn)


def _block(s, name):
    sl = {"o": slice(0, s.nocc), "v": slice(s.nocc, s.nmo)}
    p, q, r, t = (sl[c] for c in name)
    A, B = s.L[:, p, q], s.L[:, r, t]
    return (A.reshape(s.naux, -1).T @ B.reshape(s.naux, -1)).reshape(*A.shape[1:], *B.shape[1:])


def _eia(s):
    return s.mo_energy[:s.nocc, None] - s.mo_energy[None, s.nocc:]


def _mp2(s):
    e = _eia(s)
    return (_block(s, "ovov").permute(0, 2, 1, 3) / (e[:, None, :, None] + e[None, :, None, :])).contiguous()


def _binding_operands(case, seed):
    """T2 and the operand of each term: random intermediates of the
    integrals' magnitude, ovov from the factor."""
    s = _system(case, seed)
    o, v = s.nocc, s.nvir
    g = _generator(seed + 77_000_000)

    def w(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=F64) * 0.02
    ovov = _block(s, "ovov")
    Wvoov, Wvovo = w(v, o, o, v), w(v, o, v, o)
    # device tensors come in the layout this framework's own driver passes
    # (rows (c, d)); the reference's driver passes plain [a, b, c, d] arrays
    Wvvvv = w(v, v, v, v) if case["host"] else w(v, v, v, v).permute(2, 3, 0, 1)
    W = {"0101": w(o, o, o, o), "2323": Wvvvv, "1302": Wvoov, "1202": Wvovo, "1303": Wvoov, "1203": Wvovo}
    for t in ("1323", "0112", "0113", "0313", "0312"):
        W[t] = ovov
    shape = {"1323": (o, o, o, o), "0312": (v, o, v, o)}
    for t in ("0112", "0113", "0313"):
        shape[t] = (v, o, o, v)
    return s, _mp2(s), W, {t: shape.get(t, (o, o, v, v)) for t in TERMS}


def prepare(case, seed):
    kind, m = case["kind"], case["m"]
    st = SimpleNamespace(kind=kind, case=dict(case))
    if kind in ("compress", "pivotal"):
        s = _system(case, seed)
        st.x, st.rn = _mp2(s).reshape(-1), s.rn[0]
        st.hist = [int(w) for w in rng.GlibcRand(int(seed) + 1).history()]
        return st
    if kind == "binding":
        s, t2, W, st.shapes = _binding_operands(case, seed)
        st.rn = s.rn[0]
        if case["host"]:
            seen = {}
            st.W = {t: seen.setdefault(id(x), x.cpu().numpy()) for t, x in W.items()}
            st.t2 = t2.cpu().numpy()
        else:
            st.W, st.t2 = W, t2
        return st
    s = _system(case, seed)
    if kind == "build":
        st.system = s
        return st
    st.rn, st.t1, st.t2 = s.rn, s.t1, _mp2(s)
    split = case["precision"] == "split"
    eris = cholesky.split_eris(s) if split else rccsd_dense.DeviceERIs.from_system(s)
    if kind == "iterate":
        st.solver = friccsd.FRICCSDGPU(eris, {"m_keep": m}, precision=case["precision"])
    elif kind == "linear":
        st.solver = frilccsd.FRILCCSDGPU(eris, {"m_keep": m}, precision=case["precision"])
        st.rn = st.rn[:st.solver.n_draws]
    else:
        seeds = _replica_seeds(case, seed)
        st.solver = replicas.FusedReplicaBatch(eris, {"m_keep": m}, seeds, precision=case["precision"])
        R = case["replicas"]
        st.t1 = st.t1.unsqueeze(0).repeat(R, 1, 1).contiguous()
        st.t2 = st.t2.unsqueeze(0).repeat(R, 1, 1, 1, 1).contiguous()
        st.hists = [list(r.history()) for r in st.solver.rng]
    return st


def _replica_seeds(case, seed):
    return [1000 + int(seed) % 1_000_000 + r for r in range(case["replicas"])]


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(st):
    kind, m = st.kind, st.case["m"]
    if kind in ("compress", "pivotal"):
        lib = _lib.load()
        n = st.x.numel()
        flat = torch.empty(m, dtype=torch.int64, device="cuda")
        vals = torch.empty(m, dtype=F64, device="cuda")
        nd, draws = ctypes.c_int64(0), ctypes.c_int64(0)
        if kind == "compress":
            _lib.check(lib.fricc_compress(_ptr(st.x), n, m, _lib.COMPRESSION["fri"], float(st.rn), _ptr(flat),
                                          _ptr(vals), ctypes.byref(nd), _lib.cur_stream()))
        else:
            hist = (ctypes.c_uint32 * 31)(*st.hist)
            _lib.check(lib.fricc_compress_pivotal(_ptr(st.x), n, m, hist, _ptr(flat), _ptr(vals), ctypes.byref(nd),
                                                  ctypes.byref(draws), _lib.cur_stream()))
        return {"flat": flat, "vals": vals, "n_largest": nd.value, "draws": draws.value}
    if kind == "binding":
        T = py_rccsd.SparseTensor4d(st.t2, st.t2.shape, m, "fri", "systematic", rn=st.rn)
        out = {}
        for t in TERMS:
            out[t] = np.zeros(st.shapes[t]) if st.case["host"] else \
                torch.zeros(st.shapes[t], dtype=F64, device="cuda")
            py_rccsd.contract_DTSpT(st.W[t], T, out[t], t)
        return out
    if kind == "build":
        E = cholesky.split_eris(st.system)
        return {k: getattr(E, k) for k in ("oooo", "ovoo", "ovov", "oovv", "ovvv", "S0", "U", "G_t1", "ovvv_XY")}
    if kind == "replicas":
        b = st.solver
        b.t1, b.t2 = st.t1, st.t2  # every pass is the batch's first step
        for r, h in zip(b.rng, st.hists):
            r.set_history(h)
        e_norm = b.step(record=False)
        return {"t1": b.t1, "t2": b.t2, "e_norm": e_norm}
    t1, t2 = st.solver.update_amps(st.t1, st.t2, rn=st.rn if kind == "linear" else st.rn[:2])
    e, norm = st.solver.read_energy()
    return {"t1": t1, "t2": t2, "e": e, "norm": norm}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    o, v, m, naux = (float(case[k]) for k in ("o", "v", "m", "naux"))
    n, ov = (o * v) ** 2, o * v
    kind = case["kind"]
    if kind in ("compress", "pivotal"):
        return {"bytes": 8 * n + 16 * m, "flops": 3 * n}
    o3v3, o4v2 = 2 * m * ov, 2 * m * o * o
    if kind == "binding":
        w = o ** 4 + v ** 4 + 2 * n + n           # the five operands, each once
        outs = 5 * n + o ** 4 + 4 * n + n
        return {"bytes": 8 * (n + w + outs), "flops": 2 * m * v * v + 8 * o3v3 + 2 * o4v2}
    if kind == "build":
        nmo = o + v
        blocks = o ** 4 + o ** 3 * v + 2 * n + o * v ** 3
        return {"bytes": 8 * (naux * nmo * nmo + blocks + 2 * o * v ** 3), "flops": 2 * naux * blocks}
    ints = o ** 4 + o ** 3 * v + 3 * n + o * v ** 3 + v ** 4
    if kind == "linear":
        dense = 4 * o * o * v ** 3 + 4 * o ** 3 * v * v
        return {"bytes": 8 * (ints + 2 * n), "flops": 2 * m * v * v + 4 * o3v3 + o4v2 + 2 * dense}
    dense = 12 * o * o * v ** 3 + 8 * o ** 3 * v * v
    flops = 2 * m * v * v + 4 * m * ov + 6 * o3v3 + 2 * o4v2 + dense  # 2323, X/Y, six passes, 0101 and 1323
    R = case.get("replicas", 1)
    if case["precision"] == "split":  # (vv|vv) comes from the factor
        ints += naux * v * v - v ** 4
        flops += 2 * naux * v ** 4
    return {"bytes": 8 * (ints + 2 * R * n), "flops": R * flops}


# --------------------------------------------------------------------------
# the same, in 64 bits, from the reference's definitions
# --------------------------------------------------------------------------
def _select(x, m):
    """D (flat indices of the exactly kept entries), the p vector and m - |D|
    (fri_compression's get_d_largest and make_probability_vector)."""
    a = np.abs(x)
    kth = np.partition(a, a.size - m)[a.size - m]
    cand = np.flatnonzero(a >= kth)
    top = cand[np.argsort(-a[cand], kind="stable")][:m]
    ai = a[top]
    R = np.subtract.accumulate(np.concatenate([[np.add.accumulate(a)[-1]], ai]))
    ok = ((m - np.arange(m)) * ai >= R[:m] - ai) & (R[:m] > 1e-14)
    d = m if ok.all() else int(np.argmin(ok))
    p = a / R[d] * float(m - d)
    p[top[:d]] = 0.0
    return top[:d], p, m - d


def _systematic(x, m, rn):
    """(flat, vals, |D|) of a systematic FRI compression."""
    D, p, ns = _select(x, m)
    edges = np.concatenate([[0.0], np.add.accumulate(p)])
    u = np.arange(ns) * 1.0 + rn
    S = np.searchsorted(edges, u, side="right") - 1
    S[u >= edges[-1]] = 0
    with np.errstate(all="ignore"):
        return np.concatenate([D, S]), np.concatenate([x[D], x[S] / p[S]]), len(D)


def _libc_draws(seed, count):
    libc = ctypes.CDLL(None)
    libc.rand.restype = ctypes.c_int
    libc.srand(ctypes.c_uint(seed))
    return [libc.rand() / 2147483647 for _ in range(count)]


def _pivotal(x, m, seed):
    D, p, ns = _select(x, m)
    q, draws, S, a, i, used = p.tolist(), _libc_draws(seed, x.size), [], p[0].item(), 0, 0
    for j in range(1, len(q)):
        a += q[j]
        r = draws[used]
        used += 1
        if a < 1.0:
            if r < q[j] / a:
                i = j
        else:
            a -= 1.0
            if r < (1.0 - q[j]) / (1.0 - a):
                S.append(i)
                i = j
            else:
                S.append(j)
        if len(S) == ns:
            break
        if j == len(q) - 1 and abs(a - 1.0) < 1e-5:
            S.append(i)
    S = np.array(S, dtype=np.int64)
    return np.concatenate([D, S]), np.concatenate([x[D], x[S] / p[S]]), len(D), used


def _dense_t(t2, m, rn):
    """The compressed T2 as a dense tensor."""
    flat, vals, _ = _systematic(t2.reshape(-1).cpu().numpy(), m, rn)
    T = torch.zeros(t2.numel(), dtype=F64, device=t2.device)
    T.index_put_((torch.from_numpy(flat).to(t2.device),), torch.from_numpy(vals).to(t2.device), accumulate=True)
    return T.view(t2.shape)


def _sym(x):
    return x + x.permute(1, 0, 3, 2)


EINSUM = {  # the eleven terms of contract_DTSpT
    "0101": (1.0, "klij,klab->ijab"), "2323": (1.0, "abcd,ijcd->ijab"), "1302": (2.0, "akic,kjcb->ijab"),
    "1202": (-1.0, "akci,kjcb->ijab"), "1303": (1.0, "akic,kjbc->ijab"), "1203": (1.0, "bkci,kjac->ijab"),
    "1323": (1.0, "kcld,ijcd->klij"), "0112": (-0.5, "ldkc,ilda->akic"), "0113": (1.0, "ldkc,ilad->akic"),
    "0313": (-0.5, "lckd,ilad->akic"), "0312": (-0.5, "lckd,ilda->akci"),
}


def _term(name, W, T):
    c, spec = EINSUM[name]
    return c * torch.einsum(spec, W, T)


def _ccsd(s, B, t1, t2, rn, m):
    """fricc/friccsd.py:29-301 (its sum over c, d inside Wvvvv in the t1 t1
    term included), dense FP64; returns t1new, t2new."""
    ein = torch.einsum
    o = s.nocc
    fock, fov = s.fock, s.fock[:o, o:]
    eia = _eia(s)
    T, Tw = _dense_t(t2, m, rn[0]), _dense_t(t2, m, rn[1])
    ovov, ovoo, oovv, ovvv, oooo = B["ovov"], B["ovoo"], B["oovv"], B["ovvv"], B["oooo"]
    ovvo = ovov.permute(0, 1, 3, 2)
    g = 2 * ovov - ovov.permute(0, 3, 2, 1)
    go = 2 * ovoo - ovoo.permute(2, 1, 0, 3)
    tt = t2 + ein("ic,ld->ilcd", t1, t1)
    Foo0 = fock[:o, :o] + ein("kcld,ilcd->ki", g, tt)
    Fvv0 = fock[o:, o:] - ein("kcld,klad->ac", g, tt)
    Fov = fov + ein("kcld,ld->kc", g, t1)
    eo, ev = torch.diag(s.mo_energy[:o]), torch.diag(s.mo_energy[o:])
    Foo, Fvv = Foo0 - eo, Fvv0 - ev
    gv = 2 * ein("kdac,kd->ac", ovvv, t1) - ein("kcad,kd->ac", ovvv, t1)
    gl = ein("lcki,lc->ki", go, t1)
    t1n = fov - 2 * (t1 @ fov.T) @ t1 + t1 @ Fvv.T - Foo.T @ t1
    t1n = t1n + 2 * ein("kc,kica->ia", Fov, t2) - ein("kc,ikca->ia", Fov, t2) + (t1 @ Fov.T) @ t1
    t1n = t1n + 2 * ein("kcai,kc->ia", ovvo, t1) - ein("kiac,kc->ia", oovv, t1)
    t1n = t1n + 2 * ein("kdac,ikcd->ia", ovvv, t2) - ein("kcad,ikcd->ia", ovvv, t2) + t1 @ gv.T
    t1n = t1n - ein("lcki,klac->ia", go, t2) - gl.T @ t1
    x = ein("abic,jc->ijab", ovvv.permute(1, 3, 0, 2) - ein("kibc,ka->abic", oovv, t1), t1)
    t2n = _sym(x) + ovov.permute(0, 2, 1, 3)
    t2n = t2n - _sym(ein("akij,kb->ijab", ein("kcai,jc->akij", ovvo, t1) + ovoo.permute(1, 3, 0, 2), t1))
    Loo = Foo + fov @ t1.T + gl
    Lvv = Fvv - t1.T @ fov + gv
    Wo = ein("lcki,jc->klij", ovoo, t1) + ein("kclj,ic->klij", ovoo, t1) + _term("1323", ovov, Tw)
    Wo = Wo + ein("kild,jd->klij", ein("kcld,ic->kild", ovov, t1), t1) + oooo.permute(0, 2, 1, 3)
    Wa = ein("kcad,id->akic", ovvv, t1) - ein("kcli,la->akic", ovoo, t1) + ovvo.permute(2, 0, 3, 1)
    Wa = Wa + _term("0112", ovov, Tw) + _term("0313", ovov, Tw) + _term("0113", ovov, Tw)
    Wa = Wa - ein("lkci,la->akic", ein("ldkc,id->lkci", ovov, t1), t1)
    Wb = ein("kdac,id->akci", ovvv, t1) - ein("lcki,la->akci", ovoo, t1) + oovv.permute(2, 0, 3, 1)
    Wb = Wb + _term("0312", ovov, Tw) - ein("lkci,la->akci", ein("lckd,id->lkci", ovov, t1), t1)
    t2n = t2n + ein("lija,lb->ijab", ein("klij,ka->lija", Wo, t1), t1) + _term("0101", Wo, T)
    Wv = B["vvvv"].permute(0, 2, 1, 3) - ein("kdac,kb->abcd", ovvv, t1) - ein("kcbd,ka->abcd", ovvv, t1)
    t2n = t2n + Wv.sum(dim=(2, 3))[None, None] * t1[:, None, :, None] * t1[None, :, None, :]
    t2n = t2n + _term("2323", Wv, T)
    del Wv
    t2n = t2n + _sym(ein("ac,ijcb->ijab", Lvv, t2)) - _sym(ein("ki,kjab->ijab", Loo, t2))
    t2n = t2n + _sym(_term("1302", Wa, T) + _term("1202", Wb, T))
    t2n = t2n - _sym(_term("1303", Wa, T)) - _sym(_term("1203", Wb, T))
    return t1n / eia, t2n / (eia[:, None, :, None] + eia[None, :, None, :])


def _lccsd(s, B, t1, t2, rn, m):
    """fricc/frilccsd.py:27-261 with one shared compression."""
    ein = torch.einsum
    o = s.nocc
    fov = s.fock[:o, o:]
    eia = _eia(s)
    T = _dense_t(t2, m, rn[0])
    ovov, ovoo, oovv, ovvv, oooo = B["ovov"], B["ovoo"], B["oovv"], B["ovvv"], B["oooo"]
    ovvo = ovov.permute(0, 1, 3, 2)
    go = 2 * ovoo - ovoo.permute(2, 1, 0, 3)
    t1n = fov + 2 * ein("kcai,kc->ia", ovvo, t1) - ein("kiac,kc->ia", oovv, t1)
    t1n = t1n + 2 * ein("kdac,ikcd->ia", ovvv, t2) - ein("kcad,ikcd->ia", ovvv, t2) - ein("lcki,klac->ia", go, t2)
    t1n = t1n + 2 * ein("kc,kica->ia", fov, t2) - ein("kc,ikca->ia", fov, t2)
    Wa, Wb = ovvo.permute(2, 0, 3, 1), oovv.permute(2, 0, 3, 1)
    t2n = ovov.permute(0, 2, 1, 3) + _term("2323", B["vvvv"].permute(0, 2, 1, 3), T)
    t2n = t2n + _term("0101", oooo.permute(0, 2, 1, 3), T) + _sym(_term("1302", Wa, T) + _term("1202", Wb, T))
    t2n = t2n - _sym(_term("1303", Wa, T)) - _sym(_term("1203", Wb, T))
    t2n = t2n - _sym(ein("iajk,kb->ijab", ovoo, t1)) + _sym(ein("iabc,jc->ijab", ovvv.permute(0, 1, 3, 2), t1))
    return t1n / eia, t2n / (eia[:, None, :, None] + eia[None, :, None, :])


def _energy(s, B, t1, t2, linear):
    o = s.nocc
    tau = t2 if linear else t2 + torch.einsum("ia,jb->ijab", t1, t1)
    g = 2 * B["ovov"] - B["ovov"].permute(0, 3, 2, 1)
    return float(2 * (s.fock[:o, o:] * t1).sum() + (tau.permute(0, 2, 1, 3) * g).sum())


def _norm(t1, t2, t1o, t2o):
    ov = t1.numel()
    d = (t2 - t2o).permute(0, 2, 1, 3).reshape(ov, ov)
    return float(torch.sqrt(((t1 - t1o) ** 2).sum() + (torch.tril(d) ** 2).sum()))


def exact(case, seed):
    kind, m = case["kind"], case["m"]
    if kind in ("compress", "pivotal"):
        s = _system(case, seed)
        x = _mp2(s).reshape(-1).cpu().numpy()
        if kind == "compress":
            _, vals, _ = _systematic(x, m, s.rn[0])
        else:
            _, vals, _, _ = _pivotal(x, m, int(seed) + 1)
        return {"flat": None, "vals": torch.from_numpy(vals), "n_largest": None, "draws": None}
    if kind == "binding":
        s, t2, W, _ = _binding_operands(case, seed)
        T = _dense_t(t2, m, s.rn[0])
        return {t: _term(t, W[t], T) for t in TERMS}
    s = _system(case, seed)
    B = {k: _block(s, k) for k in ("oooo", "ovoo", "ovov", "oovv", "ovvv")}
    if kind == "build":
        ovvv = B["ovvv"]
        f = s.L[:, s.nocc:, s.nocc:].sum(dim=2)
        B["S0"], B["U"] = f.T @ f, ovvv.sum(dim=(1, 3))
        B["G_t1"] = 2.0 * ovvv.permute(0, 3, 1, 2) - ovvv.permute(0, 1, 3, 2)
        B["ovvv_XY"] = torch.stack([ovvv.permute(3, 1, 0, 2), ovvv.permute(1, 3, 0, 2)], dim=2)
        return B
    B["vvvv"] = _block(s, "vvvv")
    t2 = _mp2(s)
    if kind == "replicas":
        got = [_ccsd(s, B, s.t1, t2, _libc_draws(sd, 2), m) for sd in _replica_seeds(case, seed)]
        return {"t1": torch.stack([a for a, _ in got]), "t2": torch.stack([b for _, b in got]),
                "e_norm": np.array([[_energy(s, B, a, b, False), _norm(a, b, s.t1, t2)] for a, b in got])}
    linear = kind == "linear"
    t1n, t2n = (_lccsd if linear else _ccsd)(s, B, s.t1, t2, s.rn, m)
    return {"t1": t1n, "t2": t2n, "e": _energy(s, B, t1n, t2n, linear), "norm": _norm(t1n, t2n, s.t1, t2)}
