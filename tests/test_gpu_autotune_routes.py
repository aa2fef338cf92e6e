"""A tuned df64 solver times the modular product beside its own candidates
wherever an untuned one takes it, and its iterations agree with the untuned."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_tuner_times_the_modular_route(gpulib):
    from fricc_gb300 import autotune as AT
    from fricc_gb300 import rccsd_dense as D
    from fricc_gb300.batch import mp2_device
    from fricc_gb300.friccsd import FRICCSDGPU
    from fricc_gb300.synthetic import make_system
    s = make_system("o10v40", seed=1)
    E = D.DeviceERIs.from_system(s)
    t1, t2 = mp2_device(E)
    m = 20_000
    a = FRICCSDGPU(E, {"m_keep": m}, precision="df64", autotune=True)
    b = FRICCSDGPU(E, {"m_keep": m}, precision="df64")
    for it in range(3):
        rn = [0.2 + 0.2 * it, 0.55]
        a1, a2 = a.update_amps(t1, t2, rn=rn)
        b1, b2 = b.update_amps(t1, t2, rn=rn)
        torch.testing.assert_close(a2, b2, rtol=1e-12, atol=1e-16)
        t1, t2 = a1, a2
    assert gpulib.fricc_mod_mode() == -1  # every override taken back
    modular = {k for k, res in a._tuner.trials.items() if any(cfg == AT.MOD_CANDIDATE for _, cfg in res)}
    # a term an untuned solver runs as a modular product has been timed as one
    sparse = [k for k in a._tuner.trials if k[0] == "spmm"]
    taken = [k for k in sparse if D.takes_mod(k[6], m, k[1:6], True, True)]
    assert taken and set(taken) <= modular
    assert all(k in modular for k in sparse if D.takes_mod(k[6], m, k[1:6], False, True))
    for k, cfg in a._tuner.best.items():  # and kept where it was the fastest
        assert cfg == min(a._tuner.trials[k], key=lambda r: r[0])[1]
