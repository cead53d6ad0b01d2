"""Performance cases of the pulsar search: what a user's program calls, at the
sizes it calls it with.

Kinds of case (the case's "kind"):

  search      DmSearch.run of a device-resident filterbank: staging,
              dedispersion, detrend + normalise, FFA, peaks, candidates,
              harmonic flags and the fold of the best candidate.
  batch       BatchSearch.run of several observations of uneven geometry.
  dedisperse  DedispersionProgram.stage + run over every DM trial.
  preprocess  PreprocessProgram.run + normalise_inplace (running-median detrend,
              statistics, normalisation) on a dedispersed uint32 block.
  ffa         FfaProgram.prepare + search and the sorted peak list.
  fold        fold_dedispersed_spectrum of one candidate.

Sizes follow gaffa_b200.configs (plain end-to-end, survey band, wide-range
subband, batched uneven) and the coarse search of gaffa_b200.proposal, at
lengths whose passes take milliseconds to a few hundred milliseconds.
"""
import math

import numpy as np
import torch

from gaffa_b200 import batch, configs, core, search, synth

DEV = "cuda:0"
K_DM = 4148.808  # s MHz^2


def listed():
    return [
        # the smallest search: a short, narrow observation with odd sizes, where
        # launches, host steps and round trips decide
        dict(name="search_tiny", kind="search", nchans=61, nsamples=33333, tsamp=64e-6, f_low=1200.0, f_high=1500.0,
             nbits=8, ndm=19, dm_low=0.0, dm_step=2.0, pmin=0.1, pmax=1.0, npsr=1, rfi=False, algorithm="brute"),
        # the plain end-to-end search: one bright pulsar, 10^5 raw peaks
        dict(name="search_plain", kind="search", nchans=256, nsamples=131072, tsamp=64e-6, f_low=1200.0,
             f_high=1500.0, nbits=8, ndm=64, dm_low=0.0, dm_step=3.1746, pmin=0.2, pmax=2.0, npsr=-1, rfi=False,
             algorithm="brute"),
        # the survey band and DM step with weak pulsars, a slice of its DM range
        dict(name="search_survey", kind="search", nchans=2048, nsamples=524288, tsamp=64e-6, f_low=1100.0,
             f_high=1700.0, nbits=8, ndm=128, dm_low=200.0, dm_step=0.48852, pmin=0.1, pmax=10.0, npsr=3, rfi=False,
             algorithm="brute"),
        # the wide-range subband search: 2-bit packed, RFI, candidates selected on the device
        dict(name="search_wide_subband", kind="search", nchans=4096, nsamples=1048576, tsamp=81.92e-6, f_low=300.0,
             f_high=400.0, nbits=2, ndm=220, dm_low=0.0, dm_step=0.36626, pmin=0.1, pmax=10.0, npsr=2, rfi=True,
             algorithm="subband"),
        # a batch of small uneven observations: one launch per stage, graph replays
        dict(name="batch_small", kind="batch", nobs=8, seed_laws=0, log2_low=16.0, log2_high=18.0, ndm_low=64,
             ndm_high=256),
        # survey-size dedispersion: the band and DM step of the survey search
        dict(name="dedisperse_survey", kind="dedisperse", nchans=4096, nsamples=262144, tsamp=64e-6, f_low=1100.0,
             f_high=1700.0, nbits=8, ndm=256, dm_low=300.0, dm_step=0.48852, algorithm="brute"),
        # dedispersion of the plain end-to-end workload at its size
        dict(name="dedisperse_plain", kind="dedisperse", nchans=256, nsamples=262144, tsamp=64e-6, f_low=1200.0,
             f_high=1500.0, nbits=8, ndm=512, dm_low=0.0, dm_step=0.39139, algorithm="brute"),
        # two-stage subband dedispersion of packed 2-bit data, ragged DM count
        dict(name="dedisperse_subband", kind="dedisperse", nchans=4096, nsamples=524288, tsamp=81.92e-6, f_low=300.0,
             f_high=400.0, nbits=2, ndm=201, dm_low=0.0, dm_step=0.36626, algorithm="subband"),
        # detrend + normalisation of the plain workload's dedispersed block
        dict(name="preprocess_plain", kind="preprocess", nseries=512, nsamples=262144, tsamp=64e-6, sd=256.0,
             level=32768.0),
        # FFA of long series: the survey's periods and widths, many rows per task
        dict(name="ffa_survey", kind="ffa", nseries=32, nsamples=4194304, tsamp=64e-6, pmin=0.1, pmax=10.0,
             bins_min=180, bins_max=256, duty=0.1, snr=8.0),
        # FFA of the coarse search that feeds the learned proposal: few bins, odd sizes
        dict(name="ffa_coarse", kind="ffa", nseries=129, nsamples=131077, tsamp=512e-6, pmin=0.1, pmax=12.8,
             bins_min=48, bins_max=64, duty=0.1, snr=4.5),
        # folding a candidate's aligned spectrum into subint x channel x phase
        dict(name="fold_candidate", kind="fold", nchans=1024, nsamples=200003, tsamp=64e-6, f_low=1200.0,
             f_high=1500.0, dm=87.3, period=0.4713, nbin=64, tsubint=1.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "batch", "dedisperse", "dedisperse", "dedisperse", "preprocess", "ffa",
                       "ffa", "ffa", "fold"])
    if kind in ("search", "dedisperse"):
        sub = rng.random() < 0.3
        if sub:
            c = dict(kind=kind, nchans=4 * _log(rng, 64, 1024), tsamp=81.92e-6, f_low=300.0, f_high=400.0, nbits=2,
                     dm_low=0.0, dm_step=0.36626, algorithm="subband")
            n_lo = 1 << 17
        else:
            f_low, f_high = rng.choice([(1200.0, 1500.0), (1100.0, 1700.0)])
            c = dict(kind=kind, nchans=_log(rng, 48, 4096), tsamp=64e-6, f_low=f_low, f_high=f_high, nbits=8,
                     dm_low=rng.choice([0.0, rng.uniform(0.0, 300.0)]),
                     dm_step=math.exp(rng.uniform(math.log(0.25), math.log(4.0))), algorithm="brute")
            n_lo = 1 << 16
        c["nsamples"] = _log(rng, n_lo, 1 << 19)
        c["ndm"] = _log(rng, 16, 256)
        # the delay of the highest DM stays below a quarter of the observation,
        # and the case below the largest listed one's cost
        per_dm = K_DM * (c["f_low"] ** -2 - c["f_high"] ** -2) / c["tsamp"]
        dm_top = 0.25 * c["nsamples"] / per_dm
        c["dm_low"] = round(min(c["dm_low"], 0.5 * dm_top), 3)
        c["ndm"] = max(8, min(c["ndm"], int((dm_top - c["dm_low"]) / c["dm_step"])))
        if c["algorithm"] == "brute":
            c["ndm"] = max(8, min(c["ndm"], int(2.0e11 / (c["nchans"] * c["nsamples"]))))
        c["dm_step"] = round(c["dm_step"], 5)
        if kind == "search":
            t = 0.7 * c["nsamples"] * c["tsamp"]
            c.update(pmin=round(rng.uniform(0.1, 0.4), 4), npsr=rng.randint(1, 3), rfi=sub)
            c["pmax"] = round(min(10.0, max(2.0 * c["pmin"], rng.uniform(0.1, 0.4) * t)), 4)
        return c
    if kind == "batch":
        return dict(kind=kind, nobs=rng.randint(2, 8), seed_laws=rng.randint(1, 10 ** 6), log2_low=15.5,
                    log2_high=18.0, ndm_low=40, ndm_high=256)
    if kind == "preprocess":
        n = _log(rng, 1 << 16, 1 << 21)
        return dict(kind=kind, nseries=max(4, min(_log(rng, 8, 512), (1 << 27) // n)), nsamples=n, tsamp=64e-6,
                    sd=rng.choice([256.0, 1024.0]), level=rng.choice([32768.0, 524288.0]))
    if kind == "ffa":
        coarse = rng.random() < 0.3
        n = _log(rng, 1 << 15, 1 << 18) if coarse else _log(rng, 1 << 16, 1 << 22)
        tsamp = 512e-6 if coarse else rng.choice([64e-6, 81.92e-6])
        bins_min, bins_max = (48, 64) if coarse else rng.choice([(180, 256), (180, 256), (200, 260), (120, 150)])
        pmin = round(rng.uniform(0.1, 0.5), 4)
        return dict(kind=kind, nseries=max(3, min(_log(rng, 4, 256), (1 << 26) // n)), nsamples=n, tsamp=tsamp,
                    pmin=pmin, pmax=round(min(10.0, max(2.0 * pmin, rng.uniform(0.05, 0.4) * n * tsamp)), 4),
                    bins_min=bins_min, bins_max=bins_max, duty=rng.choice([0.1, 0.2]), snr=5.0 if coarse else 8.0)
    n = _log(rng, 1 << 15, 1 << 18)
    return dict(kind=kind, nchans=_log(rng, 64, 1024), nsamples=n, tsamp=64e-6, f_low=1200.0, f_high=1500.0,
                dm=round(rng.uniform(1.0, 150.0), 2), period=round(rng.uniform(0.1, 0.9), 5),
                nbin=rng.choice([32, 64, 128]), tsubint=rng.choice([0.5, 1.0, 2.0]))


# -- inputs -------------------------------------------------------------------

def _observation(case, seed, npsr):
    rng = np.random.default_rng(7_000_003 + seed)
    tobs = case["nsamples"] * case["tsamp"]
    dm_max = case["dm_low"] + case.get("ndm", 1) * case.get("dm_step", 0.0)
    pulsars = []
    if npsr < 0:  # the plain workload's bright pulsar
        pulsars = [synth.Pulsar(period=0.5, dm=float(rng.uniform(0.4, 0.6) * dm_max), duty_cycle=0.02, amplitude=1.0)]
    for _ in range(max(0, npsr)):
        p = float(math.exp(rng.uniform(math.log(case["pmin"]), math.log(case["pmax"]))))
        d = float(rng.uniform(0.01, 0.05))
        dm = case["dm_low"] + float(rng.integers(0, case["ndm"])) * case["dm_step"]
        amp = synth.folded_snr_amplitude(float(rng.uniform(15.0, 30.0)), case["nchans"], d, p, tobs, case["tsamp"])
        pulsars.append(synth.Pulsar(period=p, dm=dm, duty_cycle=d,
                                    amplitude=amp, phase=float(rng.uniform(0.0, 1.0))))
    rfi = synth.Rfi(narrowband_fraction=0.05, narrowband_hz=50.0, impulse_hz=0.1) if case.get("rfi") else synth.Rfi()
    return synth.Observation(nchans=case["nchans"], nsamples=case["nsamples"], tsamp=case["tsamp"],
                             f_low=case["f_low"], f_high=case["f_high"], nbits=case.get("nbits", 8), seed=seed,
                             pulsars=pulsars, rfi=rfi)


def _subband(case):
    """(channels per subband, DMs per nominal DM): 64 subbands, a nominal DM every 20 pc cm^-3."""
    return max(1, case["nchans"] // 64), int(math.ceil(20.0 / case["dm_step"]))


def _series(case, seed):
    """Detrended noise series with a periodic pulse in some, and their (mean, 1/sd)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, ns = case["nsamples"], case["nseries"]
    stride = (n + 3) // 4 * 4
    x = torch.zeros(ns, stride, device=DEV)
    x[:, :n].normal_(generator=g)
    rng = np.random.default_rng(9_000_001 + seed)
    period = float(math.exp(rng.uniform(math.log(case["pmin"]), math.log(case["pmax"]))))
    phase = torch.remainder(torch.arange(n, device=DEV, dtype=torch.float64) * case["tsamp"] / period, 1.0)
    pulse = torch.exp(-0.5 * ((phase - 0.5) / 0.015) ** 2).float()
    amp = 20.0 / math.sqrt(0.0376 * n)
    x[::8, :n] += amp * pulse
    y = x[:, :n].double()
    stats = torch.stack([y.mean(1), 1.0 / y.std(1, unbiased=False)], 1).contiguous()
    return x, stats


def prepare(case, seed):
    kind = case["kind"]
    if kind == "search":
        obs = _observation(case, seed, case["npsr"])
        sbc, npn = _subband(case)
        sub = case["algorithm"] == "subband"
        ds = search.DmSearch(obs.frequencies, obs.nsamples, obs.tsamp, case["dm_low"], case["dm_step"], case["ndm"],
                             case["pmin"], case["pmax"], duty_cycle_max=0.1, nbits=case["nbits"],
                             algorithm=case["algorithm"], subband_channels=sbc, ndm_per_nominal=npn,
                             device_candidates=sub, memory_budget=60 << 30)
        return dict(kind=kind, search=ds, data=core.synth_generate(obs))
    if kind == "batch":
        cfgs = _batch_configs(case)
        for i, c in enumerate(cfgs):
            c.obs.seed = seed * 1000 + i
        return dict(kind=kind, search=batch.BatchSearch(cfgs, wave_bytes=24 << 30, finish_threads=1),
                    data=[core.synth_generate(c.obs) for c in cfgs])
    if kind == "dedisperse":
        obs = _observation(case, seed, 0)
        sbc, npn = _subband(case)
        prog = core.DedispersionProgram(obs.frequencies, obs.nsamples, obs.tsamp, case["dm_low"], case["dm_step"],
                                        case["ndm"], nbits=case["nbits"], algorithm=case["algorithm"],
                                        subband_channels=sbc, ndm_per_nominal=npn)
        stride = (prog.nout + 3) // 4 * 4
        st = dict(kind=kind, prog=prog, data=core.synth_generate(obs),
                  staged=torch.empty(int(prog.info.staged_bytes), dtype=torch.uint8, device=DEV),
                  out=torch.zeros(case["ndm"], stride, dtype=torch.int32, device=DEV), workspace=None)
        if case["algorithm"] == "subband":
            st["workspace"] = torch.empty(prog.workspace_bytes(case["ndm"]), dtype=torch.uint8, device=DEV)
        return st
    if kind == "preprocess":
        pre = core.PreprocessProgram(case["nsamples"], case["tsamp"], window_seconds=1.0, min_points=101,
                                     max_series=case["nseries"])
        raw = _dedispersed(case, seed)
        return dict(kind=kind, pre=pre, raw=raw, work=torch.empty_like(raw))
    if kind == "ffa":
        plan = _plan(case)
        ffa = core.FfaProgram(plan, max_series=case["nseries"])
        x, stats = _series(case, seed)
        return dict(kind=kind, ffa=ffa, series=x, stats=stats, n=case["nseries"], snr=case["snr"],
                    prepared=torch.zeros(case["nseries"], ffa.prepared_floats, device=DEV))
    obs = _observation(dict(case, dm_low=0.0, nbits=8), seed, 0)
    obs.pulsars = [synth.Pulsar(period=case["period"], dm=case["dm"], duty_cycle=0.03, amplitude=4.0)]
    return dict(kind=kind, case=case, freq=obs.frequencies, data=core.synth_generate(obs))


def _batch_configs(case):
    return configs.batched_uneven(seed=case["seed_laws"], nobs=case["nobs"], nchans_choices=(256, 512, 1024),
                                  log2_nsamples=(case["log2_low"], case["log2_high"]),
                                  ndm_range=(case["ndm_low"], case["ndm_high"]), dm_max=300.0, max_pulsars=2)


def _plan(case):
    return core.make_riptide_ffa_plan(case["nsamples"], case["tsamp"], case["pmin"], case["pmax"],
                                      bins_min=case["bins_min"], bins_max=case["bins_max"],
                                      duty_cycle_max=case["duty"])


def _dedispersed(case, seed):
    """A dedispersed block: noise about a level with a slow baseline drift."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, ns = case["nsamples"], case["nseries"]
    stride = (n + 3) // 4 * 4
    t = torch.arange(stride, device=DEV, dtype=torch.float32) / n
    raw = torch.empty(ns, stride, dtype=torch.int32, device=DEV)
    for s in range(ns):
        x = torch.randn(stride, device=DEV, generator=g) * case["sd"] + case["level"]
        raw[s] = (x + 4.0 * case["sd"] * torch.sin(6.2832 * (3.0 * t + s / ns))).round().to(torch.int32)
    return raw


# -- one pass -----------------------------------------------------------------

# Peak and candidate lists differ in length from input to input: their columns
# come at a fixed length, zeros after the list's end, with the list's length.
PEAK_ROWS, CANDIDATE_ROWS = 1 << 15, 1 << 13


def _padded(a, rows):
    out = np.zeros(rows, np.float64 if a.dtype.kind == "f" else np.int64)
    n = min(rows, len(a))
    out[:n] = a[:n]
    return out


def _peak_columns(p):
    cols = {k: _padded(p[k], PEAK_ROWS) for k in ("dm_index", "period", "width", "phase", "shift", "bins", "snr")}
    cols["count"] = len(p)
    return cols


def _result(r):
    c = {k: _padded(r.ranked[k], CANDIDATE_ROWS) for k in ("dm", "period", "snr", "frequency_min", "frequency_max",
                                                           "peak_count")}
    found = r.fold_profile is not None
    return {"peaks": _peak_columns(r.peaks), "candidates": c,
            "harmonic": _padded(r.harmonics["is_harmonic"], CANDIDATE_ROWS), "candidate_count": len(r.ranked),
            "unique_count": len(r.unique_candidates), "profile": r.fold_profile if found else np.zeros(64),
            "exposure": r.fold_exposure if found else np.zeros(64)}


def run(state):
    kind = state["kind"]
    if kind == "search":
        return _result(state["search"].run(state["data"]))
    if kind == "batch":
        res = state["search"].run(state["data"])
        all_of = {k: np.concatenate([getattr(r, k) for r in res]) for k in ("peaks", "ranked", "harmonics")}
        return {"peaks": _peak_columns(all_of["peaks"]),
                "candidates": {k: _padded(all_of["ranked"][k], CANDIDATE_ROWS) for k in ("dm", "period", "snr")},
                "harmonic": _padded(all_of["harmonics"]["is_harmonic"], CANDIDATE_ROWS),
                "profile": np.concatenate([np.zeros(64) if r.fold_profile is None else r.fold_profile for r in res])}
    if kind == "dedisperse":
        p = state["prog"]
        staged = p.stage(state["data"], out=state["staged"])
        out = p.run(staged, out=state["out"], workspace=state["workspace"])
        return out[:, : p.nout]
    if kind == "preprocess":
        state["work"].copy_(state["raw"])  # detrending is in place: the block as dedispersion left it
        state["pre"].run(state["work"])
        series = state["work"].view(torch.float32)
        state["pre"].normalise_inplace(series, series.shape[0])
        return series[:, : state["pre"].nsamples]
    if kind == "ffa":
        f = state["ffa"]
        prepared = f.prepare(state["series"], state["n"], state["stats"], out=state["prepared"])
        rec = f.search(prepared, state["n"], state["snr"])
        return {"prepared": prepared, "peaks": _peak_columns(core.sort_peaks(f.expand(rec, 0, 0.0, 1.0)))}
    c = state["case"]
    r = core.fold_dedispersed_spectrum(state["data"], state["freq"], c["dm"], c["period"], c["tsamp"], c["nbin"],
                                       tsubint=c["tsubint"])
    return {k: r[k] for k in ("cube", "exposure", "profile", "freq_phase", "time_phase")}


# -- cost and tolerance ---------------------------------------------------------

def _nout(case):
    top = case["dm_low"] + (case["ndm"] - 1) * case["dm_step"]
    return case["nsamples"] - int(round(K_DM * top * (case["f_low"] ** -2 - case["f_high"] ** -2) / case["tsamp"]))


def _dedisp_adds(case):
    if case["algorithm"] == "brute":
        return float(case["nchans"]) * case["ndm"] * _nout(case)
    sbc, npn = _subband(case)
    nom = -(-case["ndm"] // npn)
    return float(case["nchans"]) * nom * case["nsamples"] + -(-case["nchans"] // sbc) * float(case["ndm"]) * _nout(case)


def _ffa_flops(plan):
    """Transform adds, prefix sums and a subtraction and a maximum per boxcar and phase, of one series."""
    nw = len(plan.width_trials)
    return float(sum(int(t["rows"]) * int(t["bins"]) * math.ceil(math.log2(max(2, int(t["rows"])))) +
                     int(t["rows_eval"]) * int(t["bins"]) * (1 + 2 * nw) for t in plan.tasks))


def _search_work(nchans, nbits, nsamples, ndm, adds, plan):
    return {"bytes": float(nchans) * nsamples * nbits / 8, "flops": adds + ndm * _ffa_flops(plan)}


def work(case):
    kind = case["kind"]
    if kind == "search":
        plan = core.make_riptide_ffa_plan(_nout(case), case["tsamp"], case["pmin"], case["pmax"], duty_cycle_max=0.1)
        return _search_work(case["nchans"], case["nbits"], case["nsamples"], case["ndm"], _dedisp_adds(case), plan)
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for c in _batch_configs(case):
            o = c.obs
            g = dict(nchans=o.nchans, nsamples=o.nsamples, tsamp=o.tsamp, f_low=o.f_low, f_high=o.f_high, ndm=c.ndm,
                     dm_low=c.dm_low, dm_step=c.dm_step, algorithm="brute")
            plan = core.make_riptide_ffa_plan(_nout(g), o.tsamp, c.period_min, c.period_max, bins_min=c.bins_min,
                                              bins_max=c.bins_max, duty_cycle_max=c.duty_cycle_max)
            w = _search_work(o.nchans, 8, o.nsamples, c.ndm, _dedisp_adds(g), plan)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "dedisperse":
        return {"bytes": float(case["nchans"]) * case["nsamples"] * case["nbits"] / 8 + 4.0 * case["ndm"] * _nout(case),
                "flops": _dedisp_adds(case)}
    if kind == "preprocess":
        return {"bytes": 8.0 * case["nseries"] * case["nsamples"], "flops": 8.0 * case["nseries"] * case["nsamples"]}
    if kind == "ffa":
        plan = _plan(case)
        return {"bytes": 4.0 * case["nseries"] * (case["nsamples"] + plan.prepared_floats),
                "flops": case["nseries"] * _ffa_flops(plan)}
    nsub = math.ceil(case["nsamples"] * case["tsamp"] / case["tsubint"])
    return {"bytes": float(case["nchans"]) * case["nsamples"] + 4.0 * nsub * case["nchans"] * case["nbin"],
            "flops": 3.0 * case["nchans"] * case["nsamples"]}


def tolerance(case):
    # dedispersed sums are integers
    if case["kind"] == "dedisperse":
        return "exact"
    # float32 trend at the level of the block (6e-8 x level), against residuals of the block's scatter
    if case["kind"] == "preprocess":
        return {"rel": 4.0 * 6e-8 * case["level"] / case["sd"]}
    # float32 downsampling sums and S/N; whole values (indices of peaks) the same
    if case["kind"] == "ffa":
        return {"rel": 1e-6}
    # float32 results of FP64 sums
    return {"rel": 1e-6}


# -- 64-bit results by plain torch ------------------------------------------------

def _delay(dm, f, fref, tsamp):
    x = K_DM * dm * (1.0 / (f * f) - 1.0 / (fref * fref)) / tsamp
    return np.trunc(x + np.copysign(0.5, x)).astype(np.int64)


def _shifted_sum(rows, delays, nout, valid):
    """out[d][t] = sum over rows c of rows[c][t + delays[d][c]], zero past `valid`."""
    ndm = len(delays)
    pad = int(delays.max()) + nout
    out = torch.zeros(ndm, nout, dtype=torch.int64, device=DEV)
    src = torch.zeros(pad, dtype=torch.int64, device=DEV)
    for c in range(rows.shape[0]):
        m = min(valid, pad)
        src[:m] = rows[c, :m]
        view = src.unfold(0, nout, 1)
        out += view[torch.from_numpy(delays[:, c]).to(DEV)]
    return out


def _exact_dedisperse(case, seed):
    obs = _observation(case, seed, 0)
    data = core.synth_generate(obs)
    if case["nbits"] == 2:
        data = torch.stack([(data >> (2 * j)) & 3 for j in range(4)], 2).reshape(case["nsamples"], case["nchans"])
    rows = data.t().contiguous()
    f, fref, n = obs.frequencies, obs.ref_frequency, case["nsamples"]
    dms = case["dm_low"] + np.arange(case["ndm"], dtype=np.float64) * case["dm_step"]
    nout = n - int(_delay(dms[-1], f.min(), fref, case["tsamp"]))
    if case["algorithm"] == "brute":
        delays = np.stack([_delay(d, f, fref, case["tsamp"]) for d in dms])
        return _shifted_sum(rows, delays, nout, n)
    sbc, npn = _subband(case)
    nsb = -(-case["nchans"] // sbc)
    out = torch.zeros(case["ndm"], nout, dtype=torch.int64, device=DEV)
    mid = [f[(b * sbc + min((b + 1) * sbc, case["nchans"]) - 1) // 2] for b in range(nsb)]
    for g in range(0, case["ndm"], npn):
        nominal = case["dm_low"] + float(g) * case["dm_step"]
        coarse = _delay(nominal, f, fref, case["tsamp"])[None, :]
        inter = torch.cat([_shifted_sum(rows[b * sbc:(b + 1) * sbc], coarse[:, b * sbc:(b + 1) * sbc], n, n)
                           for b in range(nsb)])
        resid = np.stack([_delay(d - nominal, np.array(mid), fref, case["tsamp"]) for d in dms[g:g + npn]])
        out[g:g + npn] = _shifted_sum(inter, resid, nout, n)
    return out


def _exact_preprocess(case, seed):
    n, ns = case["nsamples"], case["nseries"]
    x = _dedispersed(case, seed)[:, :n].double()
    window = max(1, int(math.floor(1.0 / case["tsamp"] + 0.5)))
    window += 1 - window % 2
    factor = max(1, int(window / 101.0))
    low_n = n // factor
    low = x[:, : low_n * factor].reshape(ns, low_n, factor).mean(2)
    padded = torch.nn.functional.pad(low[None], (50, 50), mode="replicate")[0]
    med = torch.stack([padded[s].unfold(0, 101, 1).median(1).values for s in range(ns)])
    pos = (torch.arange(n, device=DEV, dtype=torch.float64) - 0.5 * (factor - 1)) / factor
    lower = pos.floor().clamp(0, low_n - 1).long()
    upper = (lower + 1).clamp(max=low_n - 1)
    frac = (pos - lower).clamp(0.0, 1.0)
    for s in range(ns):
        x[s] -= (1.0 - frac) * med[s][lower] + frac * med[s][upper]
    return (x - x.mean(1, keepdim=True)) / x.std(1, unbiased=False, keepdim=True)


def _exact_prepared(case, seed):
    plan = _plan(case)
    x, stats = _series(case, seed)
    n, ns = case["nsamples"], case["nseries"]
    x = (x[:, :n].double() - stats[:, :1]) * stats[:, 1:]
    out = torch.zeros(ns, plan.prepared_floats, dtype=torch.float64, device=DEV)
    sums = torch.nn.functional.pad(x.cumsum(1), (1, 0))
    seen, off = set(), 0
    for t in plan.tasks:
        f, m = float(t["downsample_factor"]), int(t["prepared_nsamples"])
        if f in seen:
            continue
        seen.add(f)
        if f == 1.0:
            out[:, off:off + m] = x[:, :m]
        else:
            start = torch.arange(m, device=DEV, dtype=torch.float64) * f
            end = start + f
            first = start.floor().long()
            last = end.floor().clamp(max=n - 1).long()
            w0, w1 = first + 1 - start, end - last
            out[:, off:off + m] = w0 * x[:, first] + w1 * x[:, last] + sums[:, last] - sums[:, first + 1]
        off = (off + m + 3) // 4 * 4
    return {"prepared": out, "peaks": None}


def _exact_fold(case, seed):
    st = prepare(case, seed)
    data, freq = st["data"], st["freq"]
    d = _delay(case["dm"], freq, float(freq.max()), case["tsamp"])
    nout, nc, nbin = case["nsamples"] - int(d.max()), case["nchans"], case["nbin"]
    spec = torch.stack([data[int(d[c]):int(d[c]) + nout, c] for c in range(nc)], 1)
    sub = max(1, int(round(case["tsubint"] / case["tsamp"])))
    nsub = -(-nout // sub)
    step = case["tsamp"] / case["period"] * nbin
    t = torch.arange(nout, device=DEV, dtype=torch.float64)
    lo = t * step
    hi = lo + step
    row = torch.arange(nout, device=DEV) // sub * nbin
    sums = torch.zeros(nsub * nbin, nc, dtype=torch.float64, device=DEV)
    expo = torch.zeros(nsub * nbin, dtype=torch.float64, device=DEV)
    first = lo.floor()
    for k in range(int(math.ceil(step)) + 1):
        w = (torch.minimum(hi, first + k + 1) - torch.maximum(lo, first + k)).clamp(min=0.0)
        at = row + torch.remainder(first + k, nbin).long()
        expo.index_add_(0, at, w)
        sums.index_add_(0, at, spec.double() * w[:, None])
    e = expo.reshape(nsub, 1, nbin)
    cube = torch.where(e > 0, sums.reshape(nsub, nbin, nc).transpose(1, 2) / e, torch.zeros_like(e))
    weighted = (cube * e).sum(0)
    ex = e.sum(0)
    return {"cube": cube, "exposure": expo.reshape(nsub, nbin), "profile": (weighted / ex).mean(0),
            "freq_phase": weighted / ex, "time_phase": cube.mean(1)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "dedisperse":
        if _dedisp_adds(case) > 3.0e11:
            return None
        return _exact_dedisperse(case, seed)
    if kind == "preprocess":
        return _exact_preprocess(case, seed)
    if kind == "ffa":
        return _exact_prepared(case, seed)
    if kind == "fold":
        return _exact_fold(case, seed)
    # a whole search returns a thresholded, ranked list: no 64-bit value of its own
    return None
