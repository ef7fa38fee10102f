"""The autotuners time each launch once: combinations that launch the same
kernels -- routing rounds of 8 and 16 steps, the register variants where a
launch has few cells, every route_cluster -- share its time, and no winner is
picked among them."""
import numpy as np
import pytest

from mhm_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small", ["1", "0"])
def test_equal_launches_share_a_time(monkeypatch, small):
    from mhm_gb300.model import MhmGpu
    monkeypatch.setenv("MHM_CELL_SMALL", small)
    dom = synth.make_domain(12, 10, 2, l11_factor=2, seed=5)
    f = synth.make_forcing(dom, 48, seed=2)
    g = MhmGpu(dom)
    try:
        g.prepare(synth.make_eff_params(dom, seed=3), synth.ROUTING_PARAMS_DEFAULT)
        g.set_meteo(1, **f)
        s0 = g.get_state()
        t = g.autotune_ex(1, 48, [24, 48])
        ms = np.array(t["trial_ms"]).reshape(2, 3, 3)
        assert (ms > 0).all()
        assert (ms[:, :, 1] == ms[:, :, 2]).all() and t["route_sub_steps"] in (4, 8)
        if small == "1":
            assert (ms == ms[:, :1]).all() and t["cell_blocks_per_sm"] == 4
        assert t["chunk_steps"] == (24, 48)[int(np.argmin(ms.min(axis=(1, 2))))]
        g.set_launch_config(route_cluster=8)
        r = g.autotune_route(1, 48)
        assert r["route_cluster"] == 8 == g.get_launch_config()["route_cluster"]
        assert len(set(r["route_trial_ms"])) == 1 and r["route_trial_ms"][0] > 0
        s1 = g.get_state()
        for k in s0:
            assert np.array_equal(s0[k], s1[k]), k
    finally:
        g.close()


def test_without_routing():
    from mhm_gb300.model import MhmGpu
    dom = synth.make_domain(12, 10, 2, l11_factor=2, seed=5)
    f = synth.make_forcing(dom, 24, seed=2)
    g = MhmGpu(dom, proc_routing=0)
    try:
        g.prepare(synth.make_eff_params(dom, seed=3))
        g.set_meteo(1, **f)
        t = g.autotune(1, 24)
        ms = np.array(t["trial_ms"]).reshape(3, 3)
        assert (ms[:, 0] > 0).all() and (ms[:, 1:] == -1.0).all()
        assert t["route_trial_ms"] == [-1.0] * 4 and t["route_cluster"] == 0 and t["route_sub_steps"] == 8
    finally:
        g.close()
