"""The two lengths of a routing round (4 and 8 steps fetched ahead, the two
instantiations of route_flow_kernel) and different cuts of a call into chunks
give the same discharge and routing states bit for bit, the oracle's: a network
of several blocks with few and with many members, members at their own steps
with an idle one, inflow gauges that cut a link, and adaptive routing steps
shorter and longer than the model step."""
import numpy as np
import pytest

import test_gpu_inflow as inflow
import test_gpu_routing_case2 as case2
from mhm_gb300 import synth

pytestmark = pytest.mark.gpu

ROUT_KEYS = ("qOUT", "Qmod", "qTIN", "qTR")


def _context(monkeypatch, dom, n_members, sub, chunk):
    from mhm_gb300.model import MhmGpu
    monkeypatch.setenv("MHM_ROUTE_SUB", str(sub))
    if chunk:
        monkeypatch.setenv("MHM_CHUNK_BYTES", str(2 * n_members * dom.n_cells * 8 * chunk))
    else:
        monkeypatch.delenv("MHM_CHUNK_BYTES", raising=False)
    return MhmGpu(dom, n_members=n_members)


def _same(runs):
    (qa, sa), *rest = runs
    assert np.isfinite(qa).all() and qa.max() > 0
    for q, s in rest:
        assert np.array_equal(qa, q)
        for x, y in zip(sa, s):
            for k in ROUT_KEYS:
                assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("n_members", [2, 40])
def test_rounds_and_chunks(monkeypatch, n_members):
    from oracle.oracle import OracleRun
    dom = synth.make_domain(48, 48, 3, l11_factor=2, seed=4, dem_kind="fractal", ridges=1)
    ps = [synth.make_eff_params(dom, seed=3 + m) for m in range(n_members)]
    f = synth.make_forcing(dom, 150, seed=2)
    runs = []
    for sub, chunk, calls in ((4, 40, (100, 50)), (8, 40, (100, 50)), (8, 0, (150,)), (4, 0, (1, 149)), (8, 7, (3, 147))):
        g = _context(monkeypatch, dom, n_members, sub, chunk)
        try:
            assert g.get_launch_config()["route_sub_steps"] == sub
            g.prepare(ps, synth.ROUTING_PARAMS_DEFAULT)
            g.set_meteo(1, f["pre"], f["temp"], f["pet"])
            q, t = [], 1
            for n in calls:
                q.append(g.run(t, n))
                t += n
            runs.append((np.concatenate(q, axis=2), [g.get_state(m) for m in range(n_members)]))
        finally:
            g.close()
    _same(runs)
    for m in (0, n_members - 1):
        o = OracleRun(dom, ps[m], synth.ROUTING_PARAMS_DEFAULT, kind="hmath")
        assert np.array_equal(runs[0][0][m].T, o.run(f, 1, 1, 150)[0]), m


def test_members_at_their_own_steps(monkeypatch):
    import torch
    dom = synth.make_domain(32, 28, 2, l11_factor=2, seed=6)
    ps = [synth.make_eff_params(dom, seed=10 + m) for m in range(4)]
    f = synth.make_forcing(dom, 96, seed=7)
    dev = [torch.from_numpy(np.ascontiguousarray(f[k])).cuda() for k in ("pre", "temp", "pet")]
    runs = []
    for sub, chunk in ((4, 48), (8, 48), (4, 11), (8, 29)):
        g = _context(monkeypatch, dom, 4, sub, chunk)
        try:
            g.prepare(ps, synth.ROUTING_PARAMS_DEFAULT)
            g.set_meteo(1, *dev, on_device=True)
            qs = []
            for t0 in ([1, 25, -1, 49], [-1, 73, 97, 121]):
                q = np.zeros((4, len(dom.gauge_node), 48))
                g.run_members_async(t0, 48, q)
                g.sync()
                qs.append(q)
            runs.append((np.concatenate(qs, axis=2), [g.get_state(m) for m in range(4)]))
        finally:
            g.close()
    _same(runs)


@pytest.mark.parametrize("sub", ["4", "8"])
@pytest.mark.parametrize("proc_rout,cellsize,l11", [(1, 1000.0, 2), (2, 250.0, 2), (2, 3000.0, 4)])
def test_inflow_gauges(monkeypatch, proc_rout, cellsize, l11, sub):
    monkeypatch.setenv("MHM_ROUTE_SUB", sub)
    inflow.test_gpu_inflow_gauges_bitwise(proc_rout, cellsize, l11, "0", monkeypatch)


@pytest.mark.parametrize("sub", ["4", "8"])
@pytest.mark.parametrize("cellsize,l11", [(250.0, 2), (3000.0, 4)])
def test_adaptive_routing(monkeypatch, cellsize, l11, sub):
    monkeypatch.setenv("MHM_ROUTE_SUB", sub)
    case2.test_gpu_routing_case2_bitwise(cellsize, l11, "0", monkeypatch)
