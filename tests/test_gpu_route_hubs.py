"""Nodes with more upstream links than a routing thread keeps, whose links are read
by the lanes of a warp: 9 to 70 links (less than, just and more than the lanes),
several such nodes one after another and in one warp, rounds of 4 and 8 steps,
several members -- the discharge of every
node equals the oracle's sequential L11_routing bit for bit."""
import numpy as np
import pytest

import test_gpu_route_flow as rf
from mhm_gb300 import synth

pytestmark = pytest.mark.gpu


def _hubs(widths):
    """A river 0 <- 1 <- 2 ... with widths[i] further links into node i, every third of them two links long."""
    p = [i - 1 for i in range(len(widths))]
    for i, w in enumerate(widths):
        for j in range(w - (i + 1 < len(widths))):
            p.append(i)
            if j % 3 == 0:
                p.append(len(p) - 1)
    return np.array(p)


@pytest.mark.parametrize("widths,sub", [((9,), 8), ((16, 17), 4), ((24, 8, 25, 9), 8), ((41, 2, 7, 10, 33), 4), ((31, 32, 70), 8),
                                        ((12,) * 12, 8)])
def test_every_node_against_oracle(monkeypatch, widths, sub):
    from mhm_gb300.model import MhmGpu
    from oracle.oracle import OracleRun
    parents = _hubs(widths)
    up = np.bincount(parents[parents >= 0], minlength=parents.size)
    assert sorted(up[: len(widths)]) == sorted(widths) and (up > 8).any()
    monkeypatch.setattr(rf, "_parents", lambda kind, n: parents)
    dom = rf._domain("hubs", parents.size)
    ps = [synth.make_eff_params(dom, seed=5 + m) for m in range(3)]
    f = synth.make_forcing(dom, 50, seed=6)
    g = MhmGpu(dom, n_members=3)
    try:
        g.set_launch_config(route_sub_steps=sub)
        g.prepare(ps, synth.ROUTING_PARAMS_DEFAULT)
        g.set_meteo(1, **f)
        q = np.concatenate([g.run(1, 1), g.run(2, 6), g.run(8, 43)], axis=2)
    finally:
        g.close()
    for m in range(3):
        o = OracleRun(dom, ps[m], synth.ROUTING_PARAMS_DEFAULT, kind="hmath")
        assert np.array_equal(q[m].T, o.run(f, 1, 1, 50)[0]), m
