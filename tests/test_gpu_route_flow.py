"""The routing kernel at the edges of its blocks: networks of one node, one
block, one node more than a block, a river longer than several blocks (with a
tributary at every node), a node with more upstream links than a thread keeps,
several outlets and random forests -- the discharge of every node equals the
oracle's sequential L11_routing (src/mRM/mo_mrm_routing.f90:380-481) bit for
bit, over calls shorter and longer than a round of ticks, for every length of
the round.  A wait that runs out is reported, not waited for."""
import dataclasses

import numpy as np
import pytest

from mhm_gb300 import synth

pytestmark = pytest.mark.gpu


def _parents(kind: str, n: int) -> np.ndarray:
    """Downstream node of each node (0-based, -1 an outlet)."""
    rng = np.random.default_rng(n)
    i = np.arange(n)
    if kind == "chain":          # n - 1 -> ... -> 1 -> 0
        return i - 1
    if kind == "comb":           # a river 0 <- 2 <- 4 ..., a headwater at each of its nodes
        return np.where(i % 2 == 1, i - 1, i - 2).clip(-1)
    if kind == "star":           # everything drains into node 1, that into node 0
        return np.where(i == 0, -1, np.where(i == 1, 0, 1))
    p = np.array([-1] + [int(rng.integers(max(0, k - 9), k)) for k in range(1, n)])
    if kind == "forest":
        p[1:4] = -1              # four outlets
    perm = rng.permutation(n)
    out = np.full(n, -1)
    for k in range(n):
        out[perm[k]] = perm[p[k]] if p[k] >= 0 else -1
    return out


def _domain(kind: str, n: int):
    dom = synth.make_domain(1, n, 2, l11_factor=1, seed=3)
    p = _parents(kind, n)
    links = [(v + 1, p[v] + 1) for v in range(n) if p[v] >= 0]
    nl = len(links)
    from_n, to_n = np.full(n, -9999, np.int32), np.full(n, -9999, np.int32)
    for j, (f, t) in enumerate(links):
        from_n[j], to_n[j] = f, t
    perm, ro = synth.routing_order(from_n, to_n, n, n - nl)
    rng = np.random.default_rng(1)
    return dataclasses.replace(dom, from_n=from_n, to_n=to_n, net_perm=perm, r_order=ro, n_outlets=n - nl,
                               length=rng.uniform(500.0, 1500.0, nl), slope=rng.uniform(1e-4, 0.05, nl),
                               ffp_imp=rng.uniform(0.0, 0.1, nl), gauge_node=np.arange(1, n + 1, dtype=np.int32))


@pytest.mark.parametrize("kind,n,sub", [("chain", 2, 8), ("chain", 64, 8), ("chain", 65, 4), ("chain", 300, 8),
                                        ("comb", 130, 1), ("comb", 513, 16), ("star", 10, 8), ("star", 11, 8),
                                        ("star", 200, 4), ("forest", 97, 8), ("random", 700, 8)])
def test_every_node_against_oracle(kind, n, sub):
    from mhm_gb300.model import MhmGpu
    from oracle.oracle import OracleRun
    dom = _domain(kind, n)
    p = synth.make_eff_params(dom, seed=5)
    f = synth.make_forcing(dom, 50, seed=6)
    g = MhmGpu(dom)
    try:
        g.set_launch_config(route_sub_steps=sub)
        g.prepare(p, synth.ROUTING_PARAMS_DEFAULT)
        g.set_meteo(1, **f)
        q = np.concatenate([g.run(1, 1), g.run(2, 7), g.run(9, 42)], axis=2)[0]
        st = g.get_state()
    finally:
        g.close()
    o = OracleRun(dom, p, synth.ROUTING_PARAMS_DEFAULT, kind="hmath")
    q_ref, _, _ = o.run(f, 1, 1, 50)
    assert np.array_equal(q.T, q_ref)
    for k in ("qOUT", "Qmod", "qTIN", "qTR"):
        assert np.array_equal(st[k][:n], o.state[k][:n]), k


def test_wait_that_runs_out_is_reported(monkeypatch):
    """With no second look at a step that is not there yet, the blocks down a
    long river give up: the call returns an error and the device stays usable."""
    from mhm_gb300.model import MhmError, MhmGpu
    dom = _domain("chain", 300)
    f = synth.make_forcing(dom, 24, seed=6)
    p = synth.make_eff_params(dom, seed=5)
    monkeypatch.setenv("MHM_ROUTE_POLLS", "0")
    g = MhmGpu(dom)
    monkeypatch.delenv("MHM_ROUTE_POLLS")
    h = MhmGpu(dom)
    try:
        for x in (g, h):
            x.prepare(p, synth.ROUTING_PARAMS_DEFAULT)
            x.set_meteo(1, **f)
        with pytest.raises(MhmError, match=r"\(-4\)"):
            g.run(1, 24)
        assert np.isfinite(h.run(1, 24)).all()
    finally:
        g.close()
        h.close()
