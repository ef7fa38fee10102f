"""Host forcing above 64 MB reaches the device in pieces, with the cell chain
launched piece by piece: every result -- gauges, states, per-step fluxes,
aggregated outputs -- is that of the same forcing on the device, for hourly and
daily rows, calls that start within a day, one and several chunks, pinned and
pageable memory."""
import numpy as np
import pytest

from mhm_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hourly,pinned,chunk_rows,calls", [
    (True, True, 0, (49, 71)), (True, False, 50, (120,)), (False, False, 0, (5, 1339)), (False, True, 40, (1344,))])
def test_pieces_equal_device_forcing(monkeypatch, hourly, pinned, chunk_rows, calls):
    import torch
    from mhm_gb300.model import MhmGpu
    dom = synth.make_domain(240, 290, 2, l11_factor=5, seed=4)
    p = synth.make_eff_params(dom, seed=5)
    f = synth.make_forcing(dom, 120, seed=6) if hourly else synth.make_daily_forcing(dom, 56, seed=6)
    f = {k: torch.from_numpy(f[k]) for k in ("pre", "temp", "pet")}
    per_step = 8 * dom.n_cells
    res = []
    for host in (True, False):
        if chunk_rows:
            monkeypatch.setenv("MHM_CHUNK_BYTES", str(2 * per_step * chunk_rows * (1 if hourly else 24)))
        g = MhmGpu(dom, hourly=hourly)
        try:
            g.prepare(p, synth.ROUTING_PARAMS_DEFAULT)
            keep = {k: (v.pin_memory() if pinned else v) if host else v.cuda() for k, v in f.items()}
            g.set_meteo(1, **({k: v.numpy() for k, v in keep.items()} if host else keep), on_device=not host)
            g.enable_flux_state_outputs((3, 9, 21), -1, 0, 10**9, max_slots=64)
            g.set_timing(True)
            tt, out = 1, []
            for n in calls:
                out.append(g.run(tt, n))
                tt += n
            launches = g.get_timing(0)[0]
            _, fs, at = g.read_flux_state_outputs()
            res.append((launches, out + [fs, at] + list(g.get_state().values())))
        finally:
            g.close()
    assert res[0][0] > res[1][0]   # in pieces
    for i, (a, b) in enumerate(zip(res[0][1], res[1][1])):
        assert np.array_equal(a, b), i
