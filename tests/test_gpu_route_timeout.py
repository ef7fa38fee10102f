"""A routing wait that runs out is reported once by the call that synchronises
next, for synchronous and asynchronous runs; the context then takes new states
and its later launches are not held up by the one that gave up."""
import numpy as np
import pytest

from mhm_gb300 import synth
from test_gpu_route_flow import _domain

pytestmark = pytest.mark.gpu


def test_reported_once_and_usable_after(monkeypatch):
    from mhm_gb300.model import MhmError, MhmGpu
    dom = _domain("chain", 300)
    f = synth.make_forcing(dom, 48, seed=6)
    p = synth.make_eff_params(dom, seed=5)
    monkeypatch.setenv("MHM_ROUTE_POLLS", "0")
    g = MhmGpu(dom)
    try:
        g.prepare(p, synth.ROUTING_PARAMS_DEFAULT)
        g.set_meteo(1, **f)
        first = g.get_state()
        for _ in range(2):                      # each run reports its own
            with pytest.raises(MhmError, match=r"\(-4\)"):
                g.run(1, 24)
            g.sync()                            # ... once
            assert np.isfinite(g.get_state()["soilMoist"]).all()
            g.init_states()
            now = g.get_state()
            for k in ("soilMoist", "snowpack", "qTIN", "qTR", "qOUT", "Qmod"):
                assert np.array_equal(now[k], first[k]), k
        q = np.zeros((1, len(dom.gauge_node), 24))
        g.run_async(1, 24, q)
        with pytest.raises(MhmError, match=r"\(-4\)"):
            g.init_states()                     # synchronises first
        g.init_states()
    finally:
        g.close()
