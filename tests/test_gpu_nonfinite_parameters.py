"""An infinite sealed fraction times a sealed runoff of zero is NaN, as in the
oracle (src/mHM/mo_runoff.f90:248-274), in the kernel of few cells and in the one of
one thread a cell, whatever the sealed runoff; the cells beside it keep their bits."""
import numpy as np
import pytest

from mhm_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small", ["1", "0"])
@pytest.mark.parametrize("H,sm", [(3, 1), (6, 2)])
def test_infinite_sealed_fraction(monkeypatch, small, H, sm):
    from mhm_gb300.model import MhmGpu
    from oracle.oracle import OracleRun
    monkeypatch.setenv("MHM_CELL_SMALL", small)
    dom = synth.make_domain(9, 11, H, l11_factor=3, seed=2)
    p = {k: np.array(v, float) for k, v in synth.make_eff_params(dom, seed=3).items() if v is not None}
    p["fSealed"][[4, 40]] = np.inf
    p["fSealed"][[17, 80]] = -np.inf
    f = synth.make_forcing(dom, 60, seed=4)
    g = MhmGpu(dom, proc_soilmoist=sm)
    try:
        g.prepare(p, synth.ROUTING_PARAMS_DEFAULT)
        g.enable_outputs(total_runoff=True)
        g.set_meteo(1, **f)
        g.run(1, 60)
        tro = g.get_outputs()[0][:, 0]
    finally:
        g.close()
    o = OracleRun(dom, p, synth.ROUTING_PARAMS_DEFAULT, proc_sm=sm, kind="hmath")
    ref = o.run(f, 1, 1, 60, want_tro=True)[1]
    assert np.isnan(ref).any() and np.isfinite(np.delete(ref, [4, 17, 40, 80], axis=1)).all()
    np.testing.assert_array_equal(tro, ref)
