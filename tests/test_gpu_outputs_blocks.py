"""With outputs the one-thread-a-cell kernel has a variant of 3 and one of 4 blocks
an SM, chosen by the waves of blocks a launch takes: 80 members of 780 cells (62,400,
one wave of 4 blocks, two of 3) give each member's outputs, per-step fluxes,
discharge and states as it gives them alone, where 3 blocks run."""
import numpy as np
import pytest

from mhm_gb300 import synth

pytestmark = pytest.mark.gpu

STATES = ("interc", "snowpack", "sealSTW", "unsatSTW", "satSTW", "soilMoist", "qOUT", "Qmod", "qTIN", "qTR")


def _run(dom, ps, f, sm, flags):
    from mhm_gb300.model import MhmGpu
    g = MhmGpu(dom, proc_soilmoist=sm, n_members=len(ps))
    try:
        g.prepare(ps, synth.ROUTING_PARAMS_DEFAULT)
        g.set_meteo(1, **f)
        g.enable_flux_state_outputs(flags, -1, 3, 10**9, max_slots=4)
        g.enable_fluxes()
        q = [g.run(1, 31)]
        fx = list(g.get_fluxes())
        q.append(g.run(32, 22))
        fx += g.get_fluxes()
        names, fs, at = g.read_flux_state_outputs()
        return np.concatenate(q, axis=2), fx, fs, at, [g.get_state(m) for m in range(len(ps))]
    finally:
        g.close()


@pytest.mark.parametrize("H,sm,flags", [(1, 1, (1, 3, 4, 10, 11, 20)), (3, 3, None), (5, 1, None), (8, 2, None),
                                        (6, 4, (3, 9, 21))])
def test_four_blocks_equal_three(monkeypatch, H, sm, flags):
    monkeypatch.setenv("MHM_CELL_SMALL", "0")
    dom = synth.make_domain(26, 30, H, l11_factor=3, seed=3)
    M = 80
    assert 152 * 3 * 128 < M * dom.n_cells <= 152 * 4 * 128
    ps = [synth.make_eff_params(dom, seed=100 + m) for m in range(M)]
    f = synth.make_forcing(dom, 53, seed=4)
    flags = flags or [i for i in range(1, 22) if i != 18]
    q, fx, fs, at, st = _run(dom, ps, f, sm, flags)
    assert np.isfinite(q).all() and np.isfinite(fs).all() and fs.shape[0] == 2
    for m in (0, 3, 41, M - 1):
        q1, fx1, fs1, at1, st1 = _run(dom, [ps[m]], f, sm, flags)
        assert np.array_equal(at, at1) and np.array_equal(q[m], q1[0])
        assert np.array_equal(fs.reshape(fs.shape[0], fs.shape[1], M, -1)[:, :, m], fs1.reshape(fs.shape[0], fs.shape[1], -1))
        for a, b in zip(fx, fx1):
            assert np.array_equal(a.reshape(a.shape[0], M, -1)[:, m], b.reshape(a.shape[0], -1))
        for k in STATES:
            assert np.array_equal(st[m][k], st1[0][k]), k
