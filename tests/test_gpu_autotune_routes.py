"""A tuned df64 solver times the modular product beside its own candidates
wherever an untuned one takes it, and its iterations agree with the untuned."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v,m", [(6, 24, 2000), (20, 100, 200_000)])
def test_tuner_times_the_modular_route(gpulib, o, v, m):
    """At the smaller size sparse terms take that route (float pairs are the
    two arms' other one, good to ~1e-13), at the larger one dense products
    with a kept operand."""
    from fricc_gb300 import autotune as AT
    from fricc_gb300 import rccsd_dense as D
    from fricc_gb300.batch import mp2_device
    from fricc_gb300.friccsd import FRICCSDGPU
    from fricc_gb300.synthetic import DeviceSystem
    E = D.DeviceERIs.from_system(DeviceSystem(o, v, 8 * (o + v), 0.04, seed=1))
    t1, t2 = mp2_device(E)
    a = FRICCSDGPU(E, {"m_keep": m}, precision="df64", autotune=True)
    b = FRICCSDGPU(E, {"m_keep": m}, precision="df64")
    for it in range(2):
        rn = [0.2 + 0.2 * it, 0.55]
        a1, a2 = a.update_amps(t1, t2, rn=rn)
        b1, b2 = b.update_amps(t1, t2, rn=rn)
        assert float((a2 - b2).norm() / b2.norm()) < 1e-11
        t1, t2 = b1, b2
    assert gpulib.fricc_mod_mode() == -1  # every override taken back
    modular = {k for k, res in a._tuner.trials.items() if any(cfg == AT.MOD_CANDIDATE for _, cfg in res)}
    const = {t for n in E.SPLIT_BLOCKS for t in D.sparse_uses(o, v)[n]}
    taken = {k for k in a._tuner.trials if k[0] == "spmm" and D.takes_mod(k[6], m, k[1:6], k[1:6] in const, True)}
    dense = {k for k in a._tuner.trials if k[0] == "gemm" and (k[8] or k[9])
             and D.gemm_takes_mod(k[5][-2], k[5][-1], k[1][-1], bool(k[8]), bool(k[9]), True)}
    assert taken if o == 6 else dense
    assert modular == taken | dense
    for k, cfg in a._tuner.best.items():  # and it is kept where it was the fastest
        assert cfg == min(a._tuner.trials[k], key=lambda r: r[0])[1]
