"""The calls this package is used for, at the sizes it is used at, as measurable cases.

A case names one basin and one way of advancing it:

  step       a host program steps a small basin itself (the reference's
             do_time_step loop) and reads a storage back after every call
  run        run(tt0, n): consecutive time windows of one basin, forcing on
             the device or in host memory, hourly or daily; `state` says what
             the program reads afterwards besides the gauges
  outputs    run() with the daily flux/state and routed-discharge files on
  calibrate  one iteration of a calibration: MPR of new parameter vectors,
             default states, one run from step 1, the gauges of every set
  batch      basins of uneven size advanced together by MhmBatch

Passes of step / run / outputs / batch continue the simulation, as a program's
windows do; a calibration pass starts over.  Basins come from the package's own
generators (synth), with eight gauges; forcing has their distributions and is
drawn on the GPU.  exact() restates the model in plain torch, FP64.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from mhm_gb300 import params as gparams
from mhm_gb300 import synth
from mhm_gb300.model import MhmBatch, MhmGpu

OUT_FLAGS = (1, 2, 3, 5, 7, 8, 9, 10, 11, 15, 16, 21)   # storages, SWC per horizon, PET, aET, Q, QB, recharge, melt
BASE = dict(kind="run", nrows=96, ncols=96, H=3, l11=4, dem="plane", ridges=0, steps=240, daily=False, host=False,
            field="white", pet=0, sm=1, rout=1, members=1, basins=1, catalogue=21, tune=False, state="all")


def _case(name=None, **kw):
    c = dict(BASE, **kw)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one hourly step per call of a basin the size of the reference's test domain (34 cells of 24 km),
        # daily forcing handed over by the host, a storage read back: coupling to another model
        _case("coupled_step", kind="step", nrows=6, ncols=6, H=2, l11=1, steps=1, daily=True, host=True, state="sat"),
        # the same basin over a season in one call: the reference's own check cases (daily forcing, day/night)
        _case("small_season", nrows=6, ncols=6, H=2, l11=1, steps=2160, daily=True, host=True),
        # the plain drop-in: 96 x 96 cells, 3 horizons, a month of hourly steps, restart state read
        _case("plain_month", steps=720),
        # ragged grid (61 x 47 cells, blocks of 3 x 3 cut at the edges), LAI-corrected PET, soil case 4
        _case("ragged_lai", nrows=61, ncols=47, H=5, l11=3, pet=-1, sm=4),
        # daily Tmin/Tmax forcing: Hargreaves PET, Jarvis stress, adaptive routing (several passes per step)
        _case("jarvis_daily", nrows=128, ncols=160, H=4, l11=2, daily=True, host=True, pet=1, sm=3, rout=2),
        # ten days with the daily output files on
        _case("daily_outputs", kind="outputs", nrows=200, ncols=200),
        # one iteration of a one-set-at-a-time calibration
        _case("calibrate_one", kind="calibrate"),
        # one iteration of a population of 256 parameter sets, 40,000 cells each
        _case("calibrate_256", kind="calibrate", nrows=200, ncols=200, members=256, tune=True, state="none"),
        # ten basins of 1e3 .. 1.2e5 cells, 2-6 horizons, in one fused round
        _case("uneven_batch", kind="batch", basins=10, state="none"),
        # the single large domain: 1e6 cells, 6 horizons, 62,500 routing nodes, 240 hourly steps resident in HBM
        _case("large_domain", nrows=1000, ncols=1000, H=6, dem="fractal", ridges=6, field="grf", tune=True,
              state="sat"),
        # a quarter of it from pinned host forcing
        _case("host_window", nrows=500, ncols=500, H=6, dem="fractal", ridges=3, host=True, field="grf", state="sat"),
        # routing resolution = model resolution: one node per cell, a deep river network
        _case("fine_network", nrows=250, ncols=250, H=3, l11=1, dem="fractal", ridges=6, state="sat"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "season", "run", "run", "deep", "daily", "outputs", "calibrate", "ensemble", "batch"])
    nr, nc = _log(rng, 24, 400), _log(rng, 24, 400)
    H, l11 = rng.randint(2, 6), rng.randint(1 if nr * nc < 20_000 else 2, 5)
    if kind == "step":
        return _case(kind="step", nrows=rng.randint(3, 24), ncols=rng.randint(3, 24), H=H, l11=1, state="sat",
                     steps=rng.choice([1, 2, 3, 4, 6]), daily=True, host=True)
    if kind == "season":
        return _case(nrows=rng.randint(3, 14), ncols=rng.randint(3, 14), H=rng.randint(1, 3), l11=1, daily=True,
                     host=True, steps=24 * rng.randint(10, 90), sm=rng.choice([1, 2, 3, 4]))
    if kind == "run":
        return _case(nrows=nr, ncols=nc, H=rng.randint(1, 8), l11=l11, steps=rng.randint(100, 400),
                     pet=rng.choice([0, -1]), sm=rng.choice([1, 4]), field=rng.choice(["white", "grf"]))
    if kind == "deep":
        return _case(nrows=_log(rng, 50, 250), ncols=_log(rng, 50, 250), H=rng.randint(2, 4), l11=1, dem="fractal",
                     ridges=rng.randint(0, 6), steps=rng.randint(48, 240), state="sat")
    if kind == "daily":
        return _case(nrows=_log(rng, 24, 200), ncols=_log(rng, 24, 200), H=H, l11=l11, steps=24 * rng.randint(4, 14),
                     daily=True, host=True, pet=rng.choice([0, 1]), sm=rng.choice([2, 3]), rout=rng.choice([1, 2]))
    if kind == "outputs":
        return _case(kind="outputs", nrows=_log(rng, 24, 200), ncols=_log(rng, 24, 200), H=H, l11=l11,
                     steps=24 * rng.randint(2, 12))
    if kind == "calibrate":
        return _case(kind="calibrate", nrows=_log(rng, 24, 200), ncols=_log(rng, 24, 200), H=H, l11=l11,
                     steps=rng.randint(48, 300))
    if kind == "ensemble":
        return _case(kind="calibrate", nrows=_log(rng, 24, 120), ncols=_log(rng, 24, 120), H=H, l11=l11, state="none",
                     members=rng.choice([3, 8, 17, 32, 64]), steps=rng.randint(24, 160))
    return _case(kind="batch", basins=rng.randint(3, 9), catalogue=rng.randint(1, 99), steps=rng.randint(48, 300),
                 state="none")


# ---- basins: fixed by the case (the program's plan) ----

def _gauged(dom):
    """Eight gauges spread over the network, the outlet among them (fewer nodes: every node)."""
    g = np.unique(np.linspace(1, dom.n_nodes, min(8, dom.n_nodes)).round().astype(np.int32))
    g = np.unique(np.concatenate([g, dom.gauge_node])).astype(np.int32)
    return dataclasses.replace(dom, gauge_node=g)


@functools.lru_cache(maxsize=4)
def _basin(nrows, ncols, H, l11, dem, ridges):
    kw = dict(dem_kind="fractal", fractal_beta=3.0, tilt=0.0005, ridges=ridges) if dem == "fractal" else {}
    return _gauged(synth.make_domain(nrows, ncols, H, l11, seed=1, **kw))


@functools.lru_cache(maxsize=2)
def _l0(nrows, ncols, H, l11, dem, ridges):
    return synth.make_l0(_basin(nrows, ncols, H, l11, dem, ridges), 2 if nrows * ncols > 100_000 else 4, seed=4)


@functools.lru_cache(maxsize=2)
def _uneven(n, seed):
    """n basins, cell counts log-uniform in 1e3 .. 1.2e5, 2-6 horizons, each with its own fractal DEM."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(n):
        cells = math.exp(rng.uniform(math.log(1e3), math.log(1.2e5)))
        nr = int(round(math.sqrt(cells) * rng.uniform(0.8, 1.2)))
        out.append(_gauged(synth.make_domain(nr, int(round(cells / nr)), int(rng.integers(2, 7)),
                                             4 if cells > 4e4 else 2, seed=100 + i, dem_kind="fractal",
                                             fractal_beta=3.0, tilt=0.001)))
    return out


def _dom(c):
    return _basin(c["nrows"], c["ncols"], c["H"], c["l11"], c["dem"], c["ridges"])


def _doms(c):
    return _uneven(c["basins"], c["catalogue"]) if c["kind"] == "batch" else [_dom(c)]


# ---- inputs: fixed by the seed ----

def _white(dom, days, n, hourly):
    """synth.make_forcing / make_daily_forcing's distributions, drawn on the GPU."""
    N, dev = dom.n_cells, "cuda"
    doy = torch.as_tensor(synth.day_of_year(dom.jul_start, days), device=dev, dtype=torch.float64)[:, None]
    seas = 8.0 + 10.0 * torch.sin(2 * math.pi * (doy - 81) / 365.0)
    temp = seas + 3.0 * torch.randn((n, N), device=dev, dtype=torch.float64)
    f = {"temp": temp}
    if hourly:
        dry, k, th = 0.7, 0.6, 2.0
        pet = _hargreaves(seas, seas + 5, seas - 5, dom, doy) / 24.0
        f["pet"] = pet.expand(n, N).contiguous()
    else:
        dry, k, th = 0.5, 0.8, 6.0
        half = (3.0 + 6.0 * torch.rand((n, N), device=dev, dtype=torch.float64)) / 2
        f["tmin"], f["tmax"] = temp - half, temp + half
        f["pet"] = _hargreaves(temp, f["tmax"], f["tmin"], dom, doy)
    wet = torch.rand((n, N), device=dev) >= dry
    amount = torch.distributions.Gamma(torch.tensor(k, device=dev, dtype=torch.float64), 1.0 / th).sample((n, N))
    f["pre"] = torch.where(wet, amount, 0.0)
    return f


def _hargreaves(tavg, tmax, tmin, dom, doy):
    lat = torch.deg2rad(torch.as_tensor(dom.latitude, device="cuda"))[None, :]
    dr = 1 + 0.033 * torch.cos(2 * math.pi * doy / 365.0)
    dec = 0.409 * torch.sin(2 * math.pi * doy / 365.0 - 1.39)
    ws = torch.acos(torch.clamp(-torch.tan(lat) * torch.tan(dec), -1, 1))
    ra = 24 * 60 / math.pi * 0.0820 * dr * (ws * torch.sin(lat) * torch.sin(dec) +
                                           torch.cos(lat) * torch.cos(dec) * torch.sin(ws))
    return torch.clamp(0.0023 * ra * 0.408 * (tavg + 17.8) * torch.sqrt(torch.clamp(tmax - tmin, min=0.0)), min=0.0)


def _correlate(dom, f, n):
    """Precipitation where a Gaussian random field of 20-cell length scale exceeds its 70 % quantile."""
    nr, nc = dom.nrows, dom.ncols
    ky = torch.fft.fftfreq(nr, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(nc, device="cuda")[None, :]
    filt = torch.exp(-2.0 * (math.pi * 20.0) ** 2 * (kx * kx + ky * ky))
    amount = torch.distributions.Gamma(torch.tensor(0.6, device="cuda", dtype=torch.float64), 0.5)
    for t in range(n):
        g = torch.fft.irfft2(torch.fft.rfft2(torch.randn((nr, nc), device="cuda")) * filt, s=(nr, nc))
        wet = (g > g.mean() + 0.5244 * g.std()).T.reshape(-1)
        f["pre"][t] = torch.where(wet, amount.sample((nr * nc,)), 0.0)


def _forcing(c, dom, seed):
    """The forcing rows of one pass, from step 1's date: {"pre", "temp", ...}, each [rows, cells] on the GPU."""
    torch.manual_seed(seed)
    rows = -(-c["steps"] // 24) if c["daily"] else c["steps"]
    days = np.arange(rows) if c["daily"] else np.arange(rows) // 24
    f = _white(dom, days, rows, not c["daily"])
    if c["field"] == "grf":
        _correlate(dom, f, rows)
    if c["pet"] == 1:
        f.pop("pet")
    else:
        f.pop("tmin", None), f.pop("tmax", None)
    return f


ROUT2 = np.array([1.5, 0.0, 0.0, 0.0, 0.0])   # streamflow celerity [m s-1]


def _inputs(c, seed):
    """Per basin: (domain, effective parameters or None, forcing); parameter vectors of a calibration."""
    out = []
    for i, dom in enumerate(_doms(c)):
        mpr = c["kind"] == "calibrate" or dom.n_cells > 300_000
        out.append((dom, None if mpr else synth.make_eff_params(dom, seed=seed + i), _forcing(c, dom, seed + 7 * i)))
    gam = None
    if out[0][1] is None:
        gam = (gparams.random_gammas(c["members"], c["sm"], c["pet"], c["rout"], 4, seed=seed)
               if c["kind"] == "calibrate" else gparams.default_gamma(c["sm"], c["pet"], c["rout"], 4)[None])
    return out, gam


def prepare(case, seed):
    c = case
    inp, gam = _inputs(c, seed)
    st = {"c": c, "gs": [], "f": [], "gam": gam, "tt": 1}
    for dom, eff, f in inp:
        g = MhmGpu(dom, proc_soilmoist=c["sm"], proc_pet=c["pet"], proc_routing=c["rout"], hourly=not c["daily"],
                   n_members=c["members"])
        if eff is None:
            g.mpr_setup(_l0(c["nrows"], c["ncols"], c["H"], c["l11"], c["dem"], c["ridges"]))
            g.mpr(gam)
            for m in range(c["members"]):
                g.init_states(m)
        else:
            g.prepare(eff, ROUT2 if c["rout"] == 2 else synth.ROUTING_PARAMS_DEFAULT)
        if c["host"]:   # the host program's own arrays, page-locked where a window is large
            f = {k: (v.cpu().pin_memory() if v.numel() > 1 << 20 else v.cpu()) for k, v in f.items()}
            st.setdefault("keep", []).append(f)
            f = {k: v.numpy() for k, v in f.items()}
        g.set_meteo(1, **f, on_device=not c["host"])
        if c["kind"] == "outputs":
            slots = c["steps"] // 24
            g.enable_flux_state_outputs(OUT_FLAGS, -1, 0, 10**9, max_slots=slots)
            g.enable_routed_outputs(-1, 0, 10**9, max_slots=slots)
        if c["tune"]:
            torch.cuda.synchronize()
            g.autotune(1, min(c["steps"], 96))
        st["gs"].append(g)
        st["f"].append(f)
    if c["kind"] == "batch":
        st["batch"] = MhmBatch()
    torch.cuda.synchronize()
    return st


def run(state):
    c, g, n = state["c"], state["gs"][0], state["c"]["steps"]
    tt = state["tt"]
    if c["kind"] == "calibrate":
        g.mpr(state["gam"])
        for m in range(c["members"]):
            g.init_states(m)
        out = {"q": g.run(1, n)}
    elif c["kind"] == "batch":
        state["tt"] += n
        qs = [np.zeros((1, len(x.dom.gauge_node), n)) for x in state["gs"]]
        state["batch"].run_members(state["gs"], [np.array([tt], np.int32)] * len(qs), n, qs)
        for x in state["gs"]:
            x.sync()
        return {"q%d" % i: q for i, q in enumerate(qs)}
    else:
        state["tt"] += n
        g.set_meteo((tt - 1) // 24 + 1 if c["daily"] else tt, **state["f"][0], on_device=not c["host"])
        out = {"q": g.run(tt, n)}
    if c["kind"] == "outputs":
        _, fs, at = g.read_flux_state_outputs()
        qr, qat = g.read_routed_outputs()
        out.update(fs=fs, routed=qr, closed=np.concatenate([at, qat]) - tt)
    if c["state"] == "all":
        out.update(g.get_state())
    elif c["state"] == "sat":
        out["satSTW"] = g.get_variable("L1_SATSTW")
        out["Qmod"] = g.get_variable("L11_QMOD")
    return out


def work(case):
    """Forcing read once, parameters and states read and states written once per pass, gauges, restart
    fields and output files written; operations: the additions and multiplications of the process chain
    (66 and 14 a horizon per cell-step), an elementary function of about 40 for each power law and each
    wet horizon (a fifth of them), 8 per node-step of routing; MPR is small beside the steps."""
    c, b, fl = case, 0.0, 0.0
    n, M = c["steps"], c["members"]
    for dom in _doms(c):
        N, H, L, G = dom.n_cells, dom.n_horizons, dom.n_nodes, len(dom.gauge_node)
        rows = -(-n // 24) if c["daily"] else n
        b += rows * 3 * N * 8 + M * N * 8 * (17 + 5 * H + 2 * (5 + H)) + M * L * 8 * 8 + M * G * n * 8
        b += {"all": N * (5 + H) + 8 * L, "sat": N + L, "none": 0}[c["state"]] * 8
        if c["kind"] == "outputs":
            b += n // 24 * ((len(OUT_FLAGS) - 1 + H) * N + L) * 8
        fl += M * n * (N * (66 + 14 * H + 40 * (2 + 0.4 * H)) + 8.0 * L)
    return {"bytes": b, "flops": fl}


# ---- the model in plain torch, FP64 ----

def exact(case, seed):
    c = case
    if c["members"] * c["steps"] > 6000:
        return None
    inp, gam = _inputs(c, seed)
    res = []
    for dom, eff, f in inp:
        rp = ROUT2 if c["rout"] == 2 else synth.ROUTING_PARAMS_DEFAULT
        if eff is not None:
            res.append(_model(c, dom, {k: torch.as_tensor(v, device="cuda") for k, v in eff.items()}, rp, f))
            continue
        l0 = _l0(c["nrows"], c["ncols"], c["H"], c["l11"], c["dem"], c["ridges"])
        soil = _l0_tables(dom, l0)
        res.append([_model(c, dom, _mpr(dom, l0, soil, g), g[-9:-4], f) for g in gam])
    if c["kind"] == "batch":
        return {"q%d" % i: r["q"] for i, r in enumerate(res)}
    if isinstance(res[0], list):
        out = dict(res[0][0], q=torch.cat([r["q"] for r in res[0]]))
    else:
        out = res[0]
    keep = {"all": ("interc", "snowpack", "sealSTW", "unsatSTW", "satSTW", "soilMoist", "qOUT", "Qmod", "qTIN", "qTR",
                    "C1", "C2"), "sat": ("satSTW", "Qmod"), "none": ()}[c["state"]]
    more = ("fs", "routed", "closed") if c["kind"] == "outputs" else ()
    return {k: out[k] for k in ("q",) + keep + more}


def _calendar(dom, n):
    h = np.arange(n)
    d = np.datetime64("2000-01-01") + (dom.jul_start - synth.JUL_2000) + h // 24
    month = d.astype("M8[M]").astype(int) % 12
    doy = (d - d.astype("M8[Y]").astype("M8[D]")).astype(int) + 1
    return month, h % 24, doy


def _model(c, dom, p, rp, f):
    N, H, n, dev = dom.n_cells, dom.n_horizons, c["steps"], "cuda"
    f = {k: v.to(dev) for k, v in f.items()}
    eps = float(np.finfo(float).eps)
    month, hour, doy = _calendar(dom, n)
    hz = {k: p[k].reshape(H, N) for k in ("soilMoistSat", "soilMoistFC", "wiltingPoint", "soilMoistExp", "fRoots")}
    sms, fc, pw, beta, fr = (hz[k] for k in ("soilMoistSat", "soilMoistFC", "wiltingPoint", "soilMoistExp", "fRoots"))
    Z = torch.zeros(N, dtype=torch.float64, device=dev)
    interc, seal, snow, unsat, sat = Z, Z, Z + 15.0, Z + 10.0, Z + 75.0
    SM = list(0.5 * fc)
    fs, fns = p["fSealed"], 1.0 - p["fSealed"]
    c2 = dom.timestep / 24.0
    ddmax, ddnp = p["degDayMax"] * c2, p["degDayNoPre"] * c2
    ddthr = (ddmax - ddnp) / p["degDayInc"]
    k0, k1, k2, kp = (c2 / p[k] for k in ("kFastFlow", "kSlowFlow", "kBaseFlow", "kPerco"))
    lat = torch.deg2rad(torch.as_tensor(dom.latitude, device=dev))
    runoff = torch.empty((n, N), dtype=torch.float64, device=dev)
    acc = [Z] * (len(OUT_FLAGS) - 1 + H)
    fs_out = []
    W = torch.where
    for t in range(n):
        m, row = int(month[t]), t // 24 if c["daily"] else t
        if c["pet"] == 1:
            dr = 1.0 + 0.0330 * math.cos(2 * math.pi * doy[t] / 365.0)
            de = 0.4090 * math.sin(2 * math.pi * doy[t] / 365.0 - 1.39)
            om = torch.acos(torch.clamp(-torch.tan(lat) * math.tan(de), -1.0, 1.0))
            rad = 86400.0 / math.pi / 2.45e6 * 1367.0 * dr * (om * torch.sin(lat) * math.sin(de) +
                                                             torch.cos(lat) * math.cos(de) * torch.sin(om))
            dt = f["tmax"][row] - f["tmin"][row]
            pv = p["HarSamCoeff"] * rad * (f["temp"][row] + 17.8) * torch.sqrt(torch.clamp(dt, min=0.0))
            pv = p["fAsp"] * W((dt <= 0) | (f["temp"][row] <= -17.8), Z, pv)
        elif c["pet"] == -1:
            pv = p["petLAIcorFactor"].reshape(12, N)[m] * f["pet"][row]
        else:
            pv = p["fAsp"] * f["pet"][row]
        pet, temp, prec = pv, f["temp"][row], f["pre"][row]
        if c["daily"]:
            day = 6 < hour[t] <= 18
            pet = 2.0 * pet * (dom.fday_pet if day else dom.fnight_pet)[m] / 24.0
            temp = temp + (dom.fday_temp if day else dom.fnight_temp)[m]
            prec = 2.0 * prec * (dom.fday_prec if day else dom.fnight_prec)[m] / 24.0
        imax = p["maxInter"].reshape(12, N)[m]
        aux = interc + prec
        thr = torch.clamp(aux - imax, min=0.0)
        interc = torch.minimum(aux, imax)
        ec = W(imax > eps, pet * (interc / imax) ** (2.0 / 3.0), Z)
        keep = interc > ec
        ec, interc = W(keep, ec, interc), W(keep, interc - ec, Z)
        warm = temp > p["tempThresh"]
        dd = W(prec <= ddthr, ddnp + p["degDayInc"] * prec, ddmax)
        melt = W(warm, torch.minimum(dd * (temp - p["tempThresh"]), snow), Z)
        snow = W(warm, snow - melt, snow + thr)
        eff = melt + W(warm, thr, Z)
        tmp = seal + eff
        qs = W(fs > 0, torch.clamp(tmp - p["sealedThresh"], min=0.0), Z)
        ns = torch.minimum(tmp, p["sealedThresh"])
        es = torch.clamp((pet / float(dom.evap_coeff[m]) - ec) * (ns / p["sealedThresh"]), min=0.0)
        es = W(fs > 0, torch.minimum(es, ns), Z)
        seal = W(fs > 0, ns - es, seal)
        inf, above, soil_et = eff, Z, Z
        for h in range(H):
            s = SM[h]
            over_full = s > sms[h]
            frac = W(s > eps, torch.exp(beta[h] * torch.log(torch.clamp(s, min=eps) / sms[h])), Z)
            add = inf * (1.0 - frac)
            fill = s + add
            over = fill > sms[h]
            inf = W(over_full, inf, W(over, inf + (s - sms[h]), inf - add))
            s = W(over_full, s, torch.minimum(fill, sms[h]))
            e = pet - ec - above
            if c["sm"] in (1, 4):
                stress = W(s >= fc[h], fr[h], W(s > pw[h], fr[h] * (s - pw[h]) / (fc[h] - pw[h]), Z))
            else:
                th = torch.clamp((s - pw[h]) / (sms[h] - pw[h]), 0.0, 1.0)
                stress = fr[h] * torch.clamp(th / p["jarvis_thresh_c1"], max=1.0)
            e = torch.clamp(e * stress, min=0.0)
            enough = s > e
            e, s = W(enough, e, s - eps), W(enough, s - e, Z + eps)
            SM[h] = torch.clamp(s, min=eps)
            above = above + torch.clamp(e, min=0.0)
            soil_et = soil_et + e
        unsat = unsat + inf
        fast = W(unsat > p["unsatThresh"], torch.minimum(k0 * (unsat - p["unsatThresh"]), unsat - eps), Z)
        unsat = unsat - fast
        slow = W(unsat > eps, torch.minimum(k1 * torch.clamp(unsat, min=0.0) ** (1.0 + p["alpha"]), unsat - eps), Z)
        unsat = unsat - slow
        perc = kp * unsat
        rest = unsat > perc
        perc = W(rest, perc, unsat)
        sat = sat + perc * p["karstLoss"]
        unsat = W(rest, unsat - perc, Z)
        base = W(sat > 0, k2 * sat, Z)
        sat = W(sat > 0, sat - base, Z)
        runoff[t] = (base + slow + fast) * fns + qs * fs
        if c["kind"] == "outputs":
            now = [interc, snow, *SM, sum(SM) / sms.sum(0), unsat, sat, pet, soil_et * fns + ec + es * fs, runoff[t],
                   base * fns, perc * fns, melt]
            acc = [a + x for a, x in zip(acc, now)]
            if t % 24 == 23:
                mean = [a / 24.0 if i < 5 + H else a for i, a in enumerate(acc)]
                fs_out.append(torch.stack(mean))
                acc = [Z] * len(acc)
    out = {"interc": interc, "snowpack": snow, "sealSTW": seal, "unsatSTW": unsat, "satSTW": sat,
           "soilMoist": torch.cat(SM)}
    qmod, more = _routing(c, dom, rp, runoff)
    out.update(more)
    out["q"] = qmod[:, torch.as_tensor(dom.gauge_node.astype(np.int64) - 1, device=dev)].T[None].contiguous()
    if c["kind"] == "outputs":
        out["fs"] = torch.stack(fs_out)[:, :, None]
        out["routed"] = qmod.reshape(n // 24, 24, -1).mean(1)[:, None]
        out["closed"] = None
    return out


def _routing(c, dom, rp, runoff):
    """Accumulation and Muskingum routing, one diagonal (step + level) of the network at a time."""
    n, L, dev = c["steps"], dom.n_nodes, "cuda"
    nl = dom.n_links
    area = torch.as_tensor(dom.l1_area_km2, device=dev)
    node = torch.as_tensor(dom.l1_l11_id.astype(np.int64) - 1, device=dev)
    qout = torch.zeros((n, L), dtype=torch.float64, device=dev).index_add_(1, node, runoff * area) * 1000.0 / 3600.0
    C1, C2, R = np.zeros(L), np.zeros(L), 1
    if nl and c["rout"] == 1:
        K = rp[0] + rp[1] * (dom.length * 0.001) + rp[2] * dom.slope + rp[3] * dom.ffp_imp
        xi = np.clip(rp[4] * (1.0 + dom.slope / dom.slope.max()), 0.005, 0.5)
        K = np.maximum(np.minimum(K, 0.5 / xi), 0.5 / (1.0 - xi))
        C1[:nl] = 1.0 / (K * (1.0 - xi) + 0.5)
        C2[:nl] = 1.0 - C1[:nl] * K
    elif nl:
        K = dom.length / rp[0]
        given = np.array([1, 2, 3, 4, 5, 6, 10, 12, 15, 20, 30, 60, 120, 180, 240, 360, 480, 720, 1440]) * 60.0
        i = int(np.abs(given - K.min()).argmin())
        ts = given[max(i - (given[i] > K.min()), 0)]
        assert ts <= 3600.0
        R = int(round(3600.0 / ts))
        C1[:nl] = ts / (K + 0.5 * ts)
        C2[:nl] = 1.0 - C1[:nl] * K / ts
    level, frm, to = np.zeros(L, np.int64), dom.from_n[:nl].astype(int) - 1, dom.to_n[:nl].astype(int) - 1
    for i in dom.net_perm[:nl] - 1:
        level[to[i]] = max(level[to[i]], level[frm[i]] + 1)
    order = np.argsort(level, kind="stable")
    ptr = np.searchsorted(level[order], np.arange(level.max() + 2))
    down = np.full(L, L)   # a last, extra column takes what leaves the network
    down[frm] = to
    c1, c2 = np.zeros(L), np.zeros(L)
    c1[frm], c2[frm] = C1[:nl], C2[:nl]
    T = lambda a: torch.as_tensor(a, device=dev)  # noqa: E731
    o_, lev, dn, c1, c2 = T(order), T(level), T(down), T(c1), T(c2)
    S = n * R
    qin = torch.zeros((S, L + 1), dtype=torch.float64, device=dev)
    qin[:, :L] = qout.repeat_interleave(R, 0)
    in1, tr1 = torch.zeros(L, dtype=torch.float64, device=dev), torch.zeros(L, dtype=torch.float64, device=dev)
    flat = qin.view(-1)
    D = int(level.max()) + 1
    for k in range(S + D - 1):
        v = o_[ptr[max(0, k - S + 1)]:ptr[min(k, D - 1) + 1]]
        r = (k - lev[v]) * (L + 1)
        x = flat[r + v]
        q = tr1[v] + c1[v] * (in1[v] - tr1[v]) + c2[v] * (x - in1[v])
        in1[v], tr1[v] = x, q
        flat.index_add_(0, r + dn[v], q)
    qin = qin[:, :L]
    qmod = qin.reshape(n, R, L).mean(1) if R > 1 else qin
    is_link = torch.zeros(L, dtype=torch.float64, device=dev)
    is_link[T(frm)] = 1.0
    return qmod, {"qOUT": qout[-1], "Qmod": qmod[-1], "qTIN": in1.repeat(2), "qTR": (tr1 * is_link).repeat(2),
                  "C1": T(C1), "C2": T(C2)}


# mpr() for soil-moisture case 1 and aspect-corrected PET: the parameter vector's blocks
_OFF = dict(interc=0, snow=1, soil=9, runoff=26, pet=27, interflow=30, perc=35, rout=38, geo=43)


def _l0_tables(dom, l0):
    """Horizon weights of the soil database and the empirical slope distribution."""
    H, hd = dom.n_horizons, l0.horizon_depth.copy()
    Wd = np.zeros((l0.n_soil, H, l0.max_hor))
    for s in range(l0.n_soil):
        nh = l0.soil_n_hor[s]
        U, D = l0.soil_ud[s, :nh], l0.soil_ld[s, :nh]
        hd[H - 1] = l0.soil_rz_depth[s]
        for h in range(H):
            a, b = (hd[h - 1] if h else 0.0), hd[h]
            w = np.clip(np.minimum(D, b) - np.maximum(U, a), 0.0, None)
            Wd[s, h, :nh] = w / (b - a) if (w > 0).sum() > 1 else w > 0
    x = l0.slope0
    srt = np.sort(x)
    se = np.searchsorted(srt, x, side="right") / (x.size + 1.0)   # ties share the highest rank
    return Wd, hd, se


def _mpr(dom, l0, tables, gam):
    Wd, hd, se = tables
    H, N, f = dom.n_horizons, dom.n_cells, l0.factor
    blk = {k: gam[v:] for k, v in _OFF.items()}
    ps = blk["soil"]
    sand, clay, dbm = l0.soil_sand, l0.soil_clay, l0.soil_dbm
    nh, nt = l0.soil_n_hor[:, None], l0.soil_n_till[:, None]
    j = np.arange(l0.max_hor)[None]
    col = {k: np.zeros((l0.n_soil, 3) + ((H,) if i < 5 else ())) for i, k in enumerate(
        ("sms", "beta", "pw", "fc", "fr", "hl1", "k1", "alpha", "kp"))}
    last = l0.soil_rz_depth[l0.soil_id0[-1] - 1]
    for lc, pom in enumerate((ps[2] + ps[0], ps[1], ps[2])):
        till = j < nt
        db = np.where(till, 100.0 / (pom / 0.224 + (100.0 - pom) / dbm), dbm)
        ks = np.maximum(ps[12] * 10.0 ** (ps[9] + ps[10] * sand - ps[11] * clay), 1.10)
        ks = np.where(till, ks * dbm / db, ks)
        lo = sand < 66.5
        ths = np.where(lo, ps[3] + ps[4] * clay + ps[5] * db, ps[6] + ps[7] * clay + ps[8] * db)
        nn = np.where(lo, 1.392 - 0.418 * sand ** -0.024 + 1.212 * clay ** -0.704,
                      -2.562 + 7.0e-9 * sand ** 4.004 + 3.750 * clay ** -0.016)
        al = np.exp(np.where(lo, -0.648 + 0.023 * sand + 0.044 * clay - 3.168 * db,
                             -4.197 + 0.013 * sand + 0.076 * clay - 0.276 * db))
        ths, nn, al = np.clip(ths, 0.01, 1.0), np.maximum(nn, 1.01), np.maximum(al, 1e-5)
        fc = ths * np.exp(-0.60 * (2.0 + np.log10(ks)) * np.log(nn))
        pw = ths / np.maximum((1.0 + (al * 15000.0) ** nn) ** (1.0 - 1.0 / nn), 1.0)
        on = j < nh
        tot = np.where(on, ths, 0).sum(1)
        smsfc = (tot - np.where(on, fc, 0).sum(1)) / tot
        vh = np.where(on, ths * ks, 0).sum(1) / tot / ps[12]
        vv = tot / np.where(on, ths / ks, 0).sum(1) / ps[12]
        for h in range(H):
            w = np.where(on, np.maximum(Wd[:, h], 0.0), 0.0)
            bd, s1, f1, p1 = ((a * w).sum(1) for a in (db, ths, fc, pw))
            d0 = hd[h - 1] if 0 < h < H else 0.0
            d1 = l0.soil_rz_depth if h == H - 1 else np.full(l0.n_soil, hd[h])
            dr = last if h == H - 1 else hd[h]
            if h == H - 1:
                d0 = hd[H - 2]
            rc = (ps[13], ps[14], ps[13] - ps[15])[lc]
            col["sms"][:, lc, h], col["fc"][:, lc, h], col["pw"][:, lc, h] = (a * (d1 - d0) for a in (s1, f1, p1))
            col["fr"][:, lc, h] = rc ** (d0 * 0.1) - rc ** (dr * 0.1)
            col["beta"][:, lc, h] = bd * ps[16]
        pi, pp = blk["interflow"], blk["perc"]
        col["hl1"][:, lc], col["k1"][:, lc] = pi[0] * smsfc, pi[3] * (1.0 + vh)
        col["alpha"][:, lc], col["kp"][:, lc] = pi[4] / vh / (1.0 + smsfc), pp[0] * (1.0 + smsfc) / (1.0 + vv)
    # the L0 cells of every L1 cell
    nr, nc = dom.nrows, dom.ncols
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    cut = lambda a: T(a.reshape(nc, f, nr, f).transpose(0, 2, 1, 3).reshape(N, f * f))  # noqa: E731
    so, lc = cut(l0.soil_id0.astype(np.int64) - 1), cut(l0.lcover0.astype(np.int64) - 1)
    p = {}
    for name, k in (("soilMoistSat", "sms"), ("soilMoistFC", "fc"), ("wiltingPoint", "pw"), ("soilMoistExp", "beta"),
                    ("fRoots", "fr")):
        p[name] = 1.0 / torch.stack([(1.0 / T(col[k][:, :, h]))[so, lc].mean(1) for h in range(H)])
    sms, fc, pw = p["soilMoistSat"], p["soilMoistFC"], p["wiltingPoint"]
    fc = torch.where(fc > sms, 0.99 * sms, fc)
    p["wiltingPoint"], p["soilMoistFC"] = torch.where(pw > fc, 0.99 * fc, pw), fc
    p["fRoots"] = p["fRoots"] / torch.clamp(p["fRoots"], min=0.0).sum(0)
    for k in ("soilMoistSat", "soilMoistFC", "wiltingPoint", "soilMoistExp", "fRoots"):
        p[k] = p[k].reshape(-1)
    s_, pi, geo, pe = cut(se), blk["interflow"], blk["geo"], blk["pet"]
    t0 = pi[1] * (2.0 - s_)
    p["unsatThresh"] = T(col["hl1"])[so, lc].mean(1)
    k0 = torch.clamp(torch.where(lc == 0, t0 * pi[2], t0).mean(1), min=1.0)
    k1 = torch.clamp((t0 + T(col["k1"])[so, lc]).mean(1), min=2.0)
    p["kFastFlow"], p["kSlowFlow"] = torch.minimum(k0, k1), k1
    p["alpha"] = T(col["alpha"])[so, lc].mean(1)
    p["kPerco"] = torch.clamp(T(col["kp"])[so, lc].mean(1), min=2.0)
    unit = cut(l0.geo_unit0.astype(np.int64))
    near = (unit[..., None] - T(l0.geo_unit_list.astype(np.int64))).abs()
    gi = (near * 16 + torch.arange(near.shape[-1], device="cuda")).argmin(-1)   # the first of the nearest units
    p["kBaseFlow"] = torch.maximum(T(geo[:l0.n_geo])[gi].mean(1), k1)
    x, north = cut(l0.aspect0), cut(l0.y0) > 0
    low = north == (x < pe[2])
    p["fAsp"] = torch.where(low, pe[0] + pe[1] / pe[2] * x, pe[0] + pe[1] / (360.0 - pe[2]) * (360.0 - x)).mean(1)
    ff, fi = (lc == 0).double().mean(1), l0.frac_sealed_city * (lc == 1).double().mean(1)
    fp, sn, one = 1.0 - fi - ff, blk["snow"], torch.ones(N, dtype=torch.float64, device="cuda")
    p["fSealed"], p["tempThresh"], p["degDayInc"] = fi, sn[0] * one, sn[4] * one
    p["degDayNoPre"] = sn[1] * ff + (sn[1] + sn[3] + sn[2]) * fi + (sn[1] + sn[3]) * fp
    p["degDayMax"] = (sn[1] + sn[5]) * ff + (sn[1] + sn[3] + sn[2] + sn[6]) * fi + (sn[1] + sn[3] + sn[7]) * fp
    p["sealedThresh"] = blk["runoff"][0] * one
    kar = sum((unit == int(u)).double().mean(1) for u, k in zip(l0.geo_unit_list, l0.geo_unit_kar) if k)
    p["karstLoss"] = 1.0 - kar * blk["perc"][1]
    lai = T(l0.lai_lut)[cut(l0.lai_class0.astype(np.int64) - 1)]
    p["maxInter"] = (lai * blk["interc"][0]).mean(1).T.reshape(-1).contiguous()
    return p
