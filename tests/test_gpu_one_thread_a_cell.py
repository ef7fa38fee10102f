"""The kernel of one thread a cell on domains small enough for the edge cases:
launches of few cells take another kernel whatever register variant is asked
for, so MHM_CELL_SMALL=0 puts the parity scenarios -- degenerate parameters,
runoff fractions outside [0, 1], members sharing warps, every soil-moisture and
horizon case -- on cell_chain_kernel, in each of its register variants and in
the lean and the general form, against the oracle; then the blocks of 256
threads of large launches with few horizons, and the bounds-checked build."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import test_gpu_parity as parity
from mhm_gb300 import synth

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


@pytest.fixture(params=["4", "6", "8"])
def occ(request, monkeypatch):
    monkeypatch.setenv("MHM_CELL_SMALL", "0")
    monkeypatch.setenv("MHM_CELL_OCC", request.param)
    return request.param


@pytest.fixture(scope="module")
def small():
    dom = synth.make_domain(24, 32, 3, 4, seed=1)
    return dom, synth.make_eff_params(dom, seed=3), synth.make_forcing(dom, 24 * 20, seed=2)


def test_plain(occ, small):
    dom, p, f = small
    parity._assert_all_bitwise(*parity.run_pair(dom, p, f, 24 * 20, chunks=3))


@pytest.mark.parametrize("proc_sm,proc_pet", [(2, 0), (3, -1), (4, 0), (1, -1)])
def test_soil_moisture_and_pet_cases(occ, small, proc_sm, proc_pet):
    dom, p, f = small
    parity._assert_all_bitwise(*parity.run_pair(dom, p, f, 24 * 15, proc_sm=proc_sm, proc_pet=proc_pet))


@pytest.mark.parametrize("proc_sm", [1, 2])
@pytest.mark.parametrize("H", [1, 2, 4, 5, 6, 7, 8])
def test_horizons(occ, H, proc_sm):
    dom = synth.make_domain(16, 20, H, 4, seed=5)
    p = synth.make_eff_params(dom, seed=6)
    f = synth.make_forcing(dom, 24 * 10, seed=7)
    parity._assert_all_bitwise(*parity.run_pair(dom, p, f, 24 * 10, proc_sm=proc_sm))


@pytest.mark.parametrize("proc_sm", [1, 3])
def test_degenerate_parameters(occ, proc_sm):
    parity.test_degenerate_parameters_bitwise(proc_sm)


@pytest.mark.parametrize("H", [3, 6])
def test_unbounded_runoff_fraction(occ, H):
    parity.test_unbounded_runoff_fraction_bitwise(H)


def test_members_across_warps(occ):
    parity.test_members_across_warps_bitwise()


@pytest.mark.parametrize("hourly_pet", [(True, 2), (True, 3), (False, 0)])
def test_other_forcing(occ, small, hourly_pet):
    """Priestley-Taylor, Penman-Monteith and daily rows: the general form"""
    hourly, pet = hourly_pet
    dom, p, f = small
    rng = np.random.default_rng(5)
    N = dom.n_cells
    p = dict(p, PrieTayAlpha=rng.uniform(0.6, 1.2, 12 * N), aeroResist=rng.uniform(10.0, 80.0, 12 * N),
             surfResist=rng.uniform(30.0, 200.0, 12 * N))
    f = {k: v[: 24 * 10] for k, v in f.items()} if hourly else synth.make_daily_forcing(dom, 10, seed=2)
    if pet >= 2:
        f = {"pre": f["pre"], "temp": f["temp"], "netrad": rng.uniform(-20.0, 200.0, f["pre"].shape)}
    else:
        f = {k: f[k] for k in ("pre", "temp", "pet")}
    if pet == 3:
        f["eabs"], f["windspeed"] = rng.uniform(200.0, 900.0, f["pre"].shape), rng.uniform(0.5, 6.0, f["pre"].shape)
    parity._assert_all_bitwise(*parity.run_pair(dom, p, f, 24 * 10, proc_pet=pet, hourly=hourly))


@pytest.mark.parametrize("H", [1, 2, 3])
@pytest.mark.parametrize("proc_sm", [1, 3])
def test_blocks_of_256_threads(monkeypatch, H, proc_sm):
    """622,592 cells and more with 6 or 8 blocks an SM; a last block that is
    not full; equal to the blocks of 128 threads of 4 blocks an SM, which the
    tests above compare with the oracle."""
    from mhm_gb300.model import MhmGpu
    dom = synth.make_domain(789, 791, H, l11_factor=64, seed=2)
    assert dom.n_cells >= 152 * 8 * 128 * 4 and dom.n_cells % 256
    p = synth.make_eff_params(dom, seed=3)
    f = synth.make_forcing(dom, 9, seed=2)
    f["pre"][:, ::3] = 0.0
    res = []
    for occ in ("4", "6", "8"):
        monkeypatch.setenv("MHM_CELL_OCC", occ)
        g = MhmGpu(dom, proc_soilmoist=proc_sm)
        try:
            g.prepare(p, synth.ROUTING_PARAMS_DEFAULT)
            g.set_meteo(1, **f)
            res.append([g.run(1, 9)] + list(g.get_state().values()))
        finally:
            g.close()
    assert np.isfinite(res[0][0]).all()
    for r in res[1:]:
        for a, b in zip(r, res[0]):
            assert np.array_equal(a, b)


def test_members_in_blocks_of_256_threads(monkeypatch):
    """... and with 4 members a tile: 8 members of 78,100 cells"""
    from mhm_gb300.model import MhmGpu
    dom = synth.make_domain(275, 284, 2, l11_factor=25, seed=2)
    assert 8 * dom.n_cells >= 152 * 8 * 128 * 4 and dom.n_cells % 64
    ps = [synth.make_eff_params(dom, seed=3 + m) for m in range(8)]
    f = synth.make_forcing(dom, 9, seed=2)
    res = []
    for occ in ("4", "6", "8"):
        monkeypatch.setenv("MHM_CELL_OCC", occ)
        g = MhmGpu(dom, n_members=8)
        try:
            g.prepare(ps, synth.ROUTING_PARAMS_DEFAULT)
            g.set_meteo(1, **f)
            res.append([g.run(1, 9)] + [v for m in (0, 5, 7) for v in g.get_state(m).values()])
        finally:
            g.close()
    for r in res[1:]:
        for a, b in zip(r, res[0]):
            assert np.array_equal(a, b)


def test_bounds_checked_build(tmp_path, monkeypatch):
    """the scenarios of the bounds-checked build on cell_chain_kernel"""
    from mhm_gb300 import build
    import bc_scenarios
    build.build(bounds_check=True)
    out = tmp_path / "bc.npz"
    monkeypatch.setenv("MHM_CELL_SMALL", "0")
    r = subprocess.run([sys.executable, str(HERE / "bc_scenarios.py"), str(out)],
                       env=dict(os.environ, MHM_BOUNDS_CHECK="1"), capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    z = np.load(out)
    assert int(z["bounds_checked"]) == 1 and bool(z["status_clean"])
    res, status = bc_scenarios.run_all()
    assert all(s is None for s in status)
    for k, v in res.items():
        assert np.array_equal(np.asarray(v).view(np.uint64), z[k].view(np.uint64)), k
