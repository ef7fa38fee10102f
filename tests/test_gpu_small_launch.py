"""Launches of few cells run in the kernel that spreads a cell over H + 2 warps;
its results are those of the one-thread-a-cell kernel (MHM_CELL_SMALL=0) and of
the oracle bit for bit -- for every horizon count, cell counts at the edges of a
block, hourly and daily forcing (day/night and hourly weights), the PET and
soil-moisture cases, members sharing a block, members at their own steps with
an idle one, and runs cut into chunks."""
import numpy as np
import pytest

from mhm_gb300 import synth

pytestmark = pytest.mark.gpu

STATES = ("interc", "snowpack", "sealSTW", "unsatSTW", "satSTW", "soilMoist", "qOUT", "Qmod", "qTIN", "qTR")


def _params(dom, pet, seed):
    p = synth.make_eff_params(dom, seed=seed)
    N = dom.n_cells
    rng = np.random.default_rng(seed)
    p["PrieTayAlpha"] = rng.uniform(0.6, 1.2, 12 * N)
    p["aeroResist"] = rng.uniform(10.0, 80.0, 12 * N)
    p["surfResist"] = rng.uniform(30.0, 200.0, 12 * N)
    p["karstLoss"] = np.where(rng.random(N) < 0.3, 0.8, 1.0)
    return p


def _forcing(dom, pet, hourly, n):
    f = synth.make_forcing(dom, n, seed=2) if hourly else synth.make_daily_forcing(dom, n, seed=2)
    rng = np.random.default_rng(5)
    if hourly:
        f["tmin"], f["tmax"] = f["temp"] - 2.0, f["temp"] + 2.0
    f["netrad"] = rng.uniform(-20.0, 200.0, f["pre"].shape)
    f["eabs"], f["windspeed"] = rng.uniform(200.0, 900.0, f["pre"].shape), rng.uniform(0.5, 6.0, f["pre"].shape)
    use = {0: ("pet",), -1: ("pet",), 1: ("tmin", "tmax"), 2: ("netrad",), 3: ("netrad", "eabs", "windspeed")}[pet]
    return {k: f[k] for k in ("pre", "temp") + use}


def _run(monkeypatch, small, dom, ps, pet, sm, hourly, steps, weights=None):
    from mhm_gb300.model import MhmGpu
    monkeypatch.setenv("MHM_CELL_SMALL", str(small))
    monkeypatch.setenv("MHM_CHUNK_BYTES", str(2 * len(ps) * dom.n_cells * 8 * 30))
    g = MhmGpu(dom, proc_soilmoist=sm, proc_pet=pet, hourly=hourly, n_members=len(ps))
    try:
        g.prepare(ps, synth.ROUTING_PARAMS_DEFAULT)
        if weights:
            g.set_meteo_weights(**weights)
        g.set_meteo(1, **_forcing(dom, pet, hourly, steps if hourly else -(-steps // 24)))
        q = np.concatenate([g.run(1, 1), g.run(2, steps - 1)], axis=2)
        return q, [g.get_state(m) for m in range(len(ps))]
    finally:
        g.close()


@pytest.mark.parametrize("H,nr,nc,pet,sm,hourly,members", [
    (1, 1, 1, 0, 1, True, 1), (2, 4, 8, -1, 4, True, 1), (3, 3, 11, 0, 1, False, 1), (4, 5, 19, 1, 3, False, 1),
    (5, 7, 9, 2, 2, True, 1), (6, 6, 16, 3, 1, True, 3), (7, 13, 5, 1, 4, False, 4), (8, 9, 9, 0, 3, True, 2)])
def test_small_equals_one_thread_a_cell(monkeypatch, H, nr, nc, pet, sm, hourly, members):
    dom = synth.make_domain(nr, nc, H, l11_factor=2, seed=1)
    ps = [_params(dom, pet, 3 + m) for m in range(members)]
    w = None
    if H == 3:
        rng = np.random.default_rng(8)
        w = {k: rng.uniform(0.0, 0.1, (24, 12, dom.n_cells)) for k in ("pre", "pet")}
        w["temp"] = rng.uniform(0.99, 1.01, (24, 12, dom.n_cells))
    qa, sa = _run(monkeypatch, 1, dom, ps, pet, sm, hourly, 75, w)
    qb, sb = _run(monkeypatch, 0, dom, ps, pet, sm, hourly, 75, w)
    assert np.array_equal(qa, qb) and np.isfinite(qa).all()
    for x, y in zip(sa, sb):
        for k in STATES:
            assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("small", [1, 0])
@pytest.mark.parametrize("H", [2, 3, 6])
def test_against_oracle(monkeypatch, small, H):
    from oracle.oracle import OracleRun
    dom = synth.make_domain(9, 15, H, l11_factor=3, seed=2)
    p = _params(dom, 0, 4)
    q, st = _run(monkeypatch, small, dom, [p], 0, 1, True, 90)
    o = OracleRun(dom, p, synth.ROUTING_PARAMS_DEFAULT, kind="hmath")
    ref, _, _ = o.run(_forcing(dom, 0, True, 90), 1, 1, 90)
    assert np.array_equal(q[0].T, ref)
    for k, ok in (("interc", "interc"), ("snowpack", "snowpack"), ("sealSTW", "sealSTW"), ("soilMoist", "SM"),
                  ("unsatSTW", "unsat"), ("satSTW", "sat")):
        assert np.array_equal(st[0][k], o.state[ok]), k


def test_members_at_their_own_steps(monkeypatch):
    import torch
    from mhm_gb300.model import MhmGpu
    dom = synth.make_domain(5, 9, 3, l11_factor=2, seed=6)
    ps = [_params(dom, 0, 10 + m) for m in range(4)]
    f = {k: torch.from_numpy(v).cuda() for k, v in synth.make_forcing(dom, 48, seed=7).items()}
    out = []
    for small in (1, 0):
        monkeypatch.setenv("MHM_CELL_SMALL", str(small))
        g = MhmGpu(dom, n_members=4)
        try:
            g.prepare(ps, synth.ROUTING_PARAMS_DEFAULT)
            g.set_meteo(1, **f, on_device=True)
            qs = []
            for t0 in ([1, 700, -1, 49], [-1, 748, 97, 97]):
                q = np.zeros((4, len(dom.gauge_node), 48))
                g.run_members_async(t0, 48, q)
                g.sync()
                qs.append(q)
            out.append((qs, [g.get_state(m) for m in range(4)]))
        finally:
            g.close()
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)
    for a, b in zip(out[0][1], out[1][1]):
        for k in STATES:
            assert np.array_equal(a[k], b[k]), k


@pytest.mark.parametrize("flags", ["all", "few"])
@pytest.mark.parametrize("H,nr,nc,pet,sm,hourly,members", [
    (1, 1, 1, 0, 1, True, 1), (2, 4, 8, 0, 4, True, 2), (3, 3, 11, 0, 1, False, 1), (6, 7, 9, 1, 3, False, 3),
    (8, 9, 9, 0, 2, True, 2)])
def test_outputs_small_equals_one_thread_a_cell(monkeypatch, flags, H, nr, nc, pet, sm, hourly, members):
    """The running sums of the output warp, and those the other kernel keeps in
    shared memory (few planes) or in device memory (all, 8 horizons): every
    output variable over daily intervals cut by calls and chunks, a warm-up,
    a step with its own weights, and the per-step fluxes."""
    from mhm_gb300.model import MhmGpu
    dom = synth.make_domain(nr, nc, H, l11_factor=2, seed=3)
    ps = [_params(dom, pet, 20 + m) for m in range(members)]
    f = _forcing(dom, pet, hourly, 80 if hourly else 4)
    rng = np.random.default_rng(2)
    w_fs, w_sms = rng.uniform(0.0, 0.5, dom.n_cells), rng.uniform(100.0, 300.0, (H, dom.n_cells))
    res = []
    for small in (1, 0):
        monkeypatch.setenv("MHM_CELL_SMALL", str(small))
        monkeypatch.setenv("MHM_CHUNK_BYTES", str(2 * members * dom.n_cells * 8 * 30))
        g = MhmGpu(dom, proc_soilmoist=sm, proc_pet=pet, hourly=hourly, n_members=members)
        try:
            g.prepare(ps, synth.ROUTING_PARAMS_DEFAULT)
            g.set_meteo(1, **f)
            g.enable_flux_state_outputs([i for i in range(1, 22) if i != 18] if flags == "all" else (3, 9, 10, 21), -1, 5, 10**9, max_slots=5)
            g.enable_fluxes()
            g.set_output_weights(members - 1, 40, w_fs, w_sms)
            q = [g.run(1, 31)]
            fx = list(g.get_fluxes())
            q.append(g.run(32, 49))
            fx += g.get_fluxes()
            names, fs, at = g.read_flux_state_outputs()
            res.append(q + fx + [fs, at] + [g.get_state(m)[k] for m in range(members) for k in STATES])
        finally:
            g.close()
    assert res[0][6].shape[0] == 3 and np.isfinite(res[0][6]).all() and np.any(res[0][6] != 0.0)
    for i, (a, b) in enumerate(zip(*res)):
        assert np.array_equal(a, b), i


@pytest.mark.parametrize("H,nr,nc", [(2, 278, 280), (2, 278, 281), (3, 417, 281), (7, 278, 281), (6, 624, 250)])
def test_default_variant_by_size(H, nr, nc):
    """around one wave of 4, 6 and 8 blocks an SM: the variant a launch takes by
    its size gives the results of a chosen one"""
    from mhm_gb300.model import MhmGpu
    dom = synth.make_domain(nr, nc, H, l11_factor=8, seed=2)
    p = _params(dom, 0, 3)
    f = _forcing(dom, 0, True, 12)
    res = []
    for occ in (None, 4):
        g = MhmGpu(dom)
        try:
            if occ:
                g.set_launch_config(cell_blocks_per_sm=occ)
            assert g.get_launch_config()["cell_blocks_per_sm"] == 4
            g.prepare(p, synth.ROUTING_PARAMS_DEFAULT)
            g.set_meteo(1, **f)
            res.append([g.run(1, 12)] + [g.get_state()[k] for k in STATES])
        finally:
            g.close()
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("occ", ["4", "8", None])
def test_fused_variants(monkeypatch, occ):
    """both register variants of the fused launch, and the one it takes by its
    tiles, give the results of each context's own launch"""
    import torch
    from mhm_gb300.model import MhmBatch, MhmGpu
    if occ:
        monkeypatch.setenv("MHM_FUSED_OCC", occ)
    doms = [synth.make_domain(9, 17, 2, l11_factor=3, seed=1), synth.make_domain(13, 11, 6, l11_factor=2, seed=2)]
    fs = [{k: torch.from_numpy(v).cuda() for k, v in synth.make_forcing(d, 60, seed=4).items()} for d in doms]
    res = []
    for fused in (True, False):
        gs, qs = [MhmGpu(d) for d in doms], [np.zeros((1, len(d.gauge_node), 60)) for d in doms]
        try:
            for g, d, f in zip(gs, doms, fs):
                g.prepare(_params(d, 0, 7), synth.ROUTING_PARAMS_DEFAULT)
                g.set_meteo(1, **f, on_device=True)
            t0 = [np.array([1], np.int32)] * 2
            if fused:
                MhmBatch().run_members(gs, t0, 60, qs)
            else:
                for g, q in zip(gs, qs):
                    g.run_members_async(t0[0], 60, q)
            for g in gs:
                g.sync()
            res.append(qs + [g.get_state()[k] for g in gs for k in STATES])
        finally:
            for g in gs:
                g.close()
    for a, b in zip(*res):
        assert np.array_equal(a, b)
