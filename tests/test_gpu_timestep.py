"""Model time steps above one hour with daily forcing: a forcing row then covers
24 steps, that is several days, so the day of year turns inside a row -- at
midnight, where neither the row, the month nor the day/night flag changes.  The
kernel of few cells and the one-thread-a-cell kernel (MHM_CELL_SMALL=0) give the
same bits, the oracle's for PET input and within 1e-12 of it (of a value, or of
the largest of its kind where a difference leaves a small one) for
Hargreaves-Samani, whose radiation term takes CUDA's trigonometric functions."""
import numpy as np
import pytest

from mhm_gb300 import synth

pytestmark = pytest.mark.gpu

STATES = {"interc": "interc", "snowpack": "snowpack", "sealSTW": "sealSTW", "unsatSTW": "unsat", "satSTW": "sat",
          "soilMoist": "SM", "qOUT": "qOUT", "Qmod": "Qmod", "qTIN": "qTIN", "qTR": "qTR"}


@pytest.mark.parametrize("pet,keys", [(1, ("pre", "temp", "tmin", "tmax")), (0, ("pre", "temp", "pet"))])
@pytest.mark.parametrize("timestep", [1, 2, 3, 4, 6, 12, 24])
def test_daily_forcing_at_any_step(monkeypatch, timestep, pet, keys):
    from mhm_gb300.model import MhmGpu
    from oracle.oracle import OracleRun
    days = 40
    steps = days * 24 // timestep
    # from a month's middle: days turn inside a row and a month
    dom = synth.make_domain(9, 13, 3, l11_factor=3, seed=4, timestep=timestep, jul_start=synth.JUL_2000 + 100)
    p = synth.make_eff_params(dom, seed=5)
    fd = synth.make_daily_forcing(dom, -(-steps // 24), seed=6)
    f = {k: fd[k] for k in keys}
    res = []
    for small in (1, 0):
        monkeypatch.setenv("MHM_CELL_SMALL", str(small))
        g = MhmGpu(dom, proc_pet=pet, hourly=False)
        try:
            g.prepare(p, synth.ROUTING_PARAMS_DEFAULT)
            g.enable_outputs(total_runoff=True)
            g.set_meteo(1, **f)
            q = g.run(1, steps)[0].T
            res.append((q, g.get_outputs()[0][:, 0], g.get_state()))
        finally:
            g.close()
    (qa, ta, sa), (qb, tb, sb) = res
    assert np.isfinite(qa).all() and qa.max() > 0
    assert np.array_equal(ta, tb) and np.array_equal(qa, qb)
    for k in STATES:
        assert np.array_equal(sa[k], sb[k]), k
    o = OracleRun(dom, p, synth.ROUTING_PARAMS_DEFAULT, proc_pet=pet, hourly=False)
    q_o, t_o, _ = o.run(f, 1, 1, steps, want_tro=True)
    for a, b in [(qa, q_o), (ta, t_o)] + [(sa[k], o.state[ko]) for k, ko in STATES.items()]:
        a, b = a.reshape(-1), np.asarray(b).reshape(-1)[: a.size]
        if pet == 1:
            np.testing.assert_allclose(a, b, rtol=1e-12, atol=1e-12 * np.abs(b).max())
        else:
            assert np.array_equal(a, b)
