"""A context chooses its register variant and routing round launch by launch until
they are set or tuned, and that state can be read and written back: reading the
configuration and writing it, or setting only another knob, leaves both choices
to the launches; a value that was set or tuned stays until 0 is written."""
import ctypes as C

import numpy as np
import pytest

from mhm_gb300 import _lib, synth

pytestmark = pytest.mark.gpu


def _raw(g):
    cfg = _lib.LaunchConfig()
    assert g.L.mhm_get_launch_config(g.ctx, C.byref(cfg)) == 0
    return cfg, (cfg.cell_blocks_per_sm, cfg.route_sub_steps, cfg.chunk_steps, cfg.route_cluster)


def test_round_trips_and_pins():
    from mhm_gb300.model import MhmError, MhmGpu
    dom = synth.make_domain(8, 8, 2, l11_factor=2, seed=5)
    g = MhmGpu(dom)
    try:
        assert _raw(g)[1] == (0, 0, 0, 0)
        assert g.L.mhm_set_launch_config(g.ctx, C.byref(_raw(g)[0])) == 0      # get -> set -> get, C
        assert _raw(g)[1] == (0, 0, 0, 0)
        was = g.get_launch_config()
        assert was["by_launch"] == ("cell_blocks_per_sm", "route_sub_steps")
        g.set_launch_config(**was)                                             # ... and Python
        assert g.get_launch_config() == was and _raw(g)[1] == (0, 0, 0, 0)
        g.set_launch_config(chunk_steps=24)                                    # another knob alone
        assert _raw(g)[1] == (0, 0, 24, 0)
        g.set_launch_config(cell_blocks_per_sm=6)
        assert _raw(g)[1] == (6, 0, 0, 0) and g.get_launch_config()["by_launch"] == ("route_sub_steps",)
        saved = g.get_launch_config()
        g.set_launch_config(cell_blocks_per_sm=4, route_sub_steps=8, chunk_steps=5)
        assert g.get_launch_config() == {"cell_blocks_per_sm": 4, "route_sub_steps": 8, "chunk_steps": 5,
                                         "route_cluster": 0}
        g.set_launch_config(**saved)
        assert _raw(g)[1] == (6, 0, 0, 0)
        for bad in ({"cell_blocks_per_sm": 5}, {"cell_blocks_per_sm": -4}, {"route_sub_steps": -1},
                    {"route_sub_steps": 17}, {"chunk_steps": -1}, {"route_cluster": 3}):
            with pytest.raises(MhmError):
                g.set_launch_config(**bad)
        with pytest.raises(ValueError):
            g.set_launch_config(by_launch=("chunk_steps",))
        assert _raw(g)[1] == (6, 0, 0, 0)
    finally:
        g.close()


def test_tuned_values_stay_and_can_be_given_back():
    from mhm_gb300.model import MhmGpu
    dom = synth.make_domain(8, 8, 2, l11_factor=2, seed=5)
    f = synth.make_forcing(dom, 24, seed=2)
    g = MhmGpu(dom)
    try:
        g.prepare(synth.make_eff_params(dom, seed=3), synth.ROUTING_PARAMS_DEFAULT)
        g.set_meteo(1, **f)
        t = g.autotune(1, 24)
        occ, sub = _raw(g)[1][:2]
        assert (occ, sub) == (t["cell_blocks_per_sm"], t["route_sub_steps"]) and occ in (4, 6, 8) and sub in (4, 8, 16)
        assert "by_launch" not in g.get_launch_config()
        q = g.run(1, 24)
        g.set_launch_config()
        assert _raw(g)[1] == (0, 0, 0, 0)
        g.init_states()
        assert np.array_equal(q, g.run(1, 24))
    finally:
        g.close()
