"""The parameter regionalisation gives a cell several warps (a horizon, a group
of means or a group of LAI entries each) and a table row 16 lanes: bit for bit
the oracle's values for cell counts at the edges of a block of 32, the fewest
and the most horizons, every PET process with class and gridded LAI, and
partly empty cells."""
import numpy as np
import pytest

from mhm_gb300 import params, synth
from mhm_gb300.model import MhmGpu
from test_mpr import _gpu_vs_oracle

pytestmark = pytest.mark.gpu

PET23 = {2: [("PriestleyTaylorCoeff", 0.75, 1.75, 1.19, 1), ("PriestleyTaylorLAIcorr", -0.5, 0.2, 0.058, 1)],
         3: [("canopyheigth_forest", 15.0, 40.0, 15.0, 1), ("canopyheigth_impervious", 0.01, 0.5, 0.02, 1),
             ("canopyheigth_pervious", 0.1, 5.0, 0.11, 1), ("displacementheight_coeff", 0.5, 0.85, 0.64, 1),
             ("roughnesslength_momentum_coeff", 0.09, 0.16, 0.095, 1),
             ("roughnesslength_heat_coeff", 0.07, 0.13, 0.075, 1), ("stomatal_resistance", 10.0, 200.0, 56.0, 1)]}


@pytest.mark.parametrize("sm,pet,H,nr,nc,factor,holes,members,gridded", [
    (1, 0, 2, 1, 31, 3, 0.0, 1, False), (4, 1, 8, 4, 8, 2, 0.2, 2, False), (2, -1, 5, 3, 11, 5, 0.3, 5, False),
    (3, 2, 4, 8, 8, 3, 0.1, 2, False), (1, 3, 3, 13, 5, 4, 0.0, 1, False), (1, 1, 7, 5, 13, 1, 0.0, 2, True),
    (4, 2, 2, 11, 3, 2, 0.1, 1, True), (2, 3, 6, 7, 9, 3, 0.0, 2, True)])
def test_edges(monkeypatch, sm, pet, H, nr, nc, factor, holes, members, gridded):
    for k, v in PET23.items():
        monkeypatch.setitem(params.PET, k, v)
    _gpu_vs_oracle(sm, pet, H=H, nr=nr, nc=nc, factor=factor, holes=holes, n_members=members, gridded=gridded)


@pytest.mark.parametrize("H,nr,nc,rout,members", [(1, 1, 1, 1, 1), (3, 15, 17, 1, 3), (8, 16, 16, 0, 2), (2, 1, 257, 1, 2)])
def test_initial_states(H, nr, nc, rout, members):
    """init_states sets one member's planes and routing states and no other's"""
    dom = synth.make_domain(nr, nc, H, l11_factor=1, seed=3)
    g = MhmGpu(dom, proc_routing=rout, n_members=members)
    try:
        rng = np.random.default_rng(1)
        old = []
        for m in range(members):
            s = {k: rng.uniform(1.0, 9.0, v.shape) for k, v in g.get_state(m).items()}
            g.set_state(s, m)
            old.append(g.get_state(m))
        g.init_states(members - 1)
        for m in range(members - 1):
            for k, v in g.get_state(m).items():
                assert np.array_equal(v, old[m][k]), k
        st = g.get_state(members - 1)
        hd = np.asarray(dom.horizon_depth, np.float64)
        top = np.concatenate([[0.0], hd])[:H]
        depth = np.concatenate([hd[:H - 1], [1500.0]])
        want = dict(interc=0.0, snowpack=15.0, sealSTW=0.0, unsatSTW=10.0, satSTW=75.0)
        for k, v in want.items():
            assert np.all(st[k] == v), k
        assert np.array_equal(st["soilMoist"].reshape(H, -1), np.repeat(((depth - top) * 0.25)[:, None], nr * nc, 1))
        for k in ("qOUT", "Qmod", "qTIN", "qTR"):
            assert rout == 0 or np.all(st[k] == 0.0), k
    finally:
        g.close()
