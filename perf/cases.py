"""Performance cases of the box and transit searches and the proposal network.

Each case is one call (or one training step) that a user's program makes through
the package's public entry points, over the range of sizes the package serves:
a quick look at a short curve up to packed batches, four-year baselines and the
network's training step.  ``listed`` names the cases that are timed, ``draw``
makes more of the same ranges, ``prepare`` / ``run`` are what a program holds
and calls, ``work`` is the least one pass has to move and compute, and ``exact``
is what the pass returns in 64-bit arithmetic, in plain torch.
"""

from __future__ import annotations

import math
import os

import numpy as np
import torch

import cuperiod_b200
from cuperiod_b200 import (BLSSettings, GridSpec, LightCurve, batch_periodograms, periodogram,
                           synthetic)
from cuperiod_b200.core import bls_power, bls_power_many
from cuperiod_b200.lightcurve import Domain, MultiBandLightCurve
from cuperiod_b200.multiband import bls_multiband_power, multiband_default_grid
from cuperiod_b200.bls import BLSMethod
from cuperiod_b200.proposal import (CHANNELS, HIDDEN, IN_CHANNELS, N_BINS, N_CLASSES, N_CONV, WIDTH,
                                    ProposalNet, Weights)
from cuperiod_b200.settings import TLSSettings
from cuperiod_b200.tls import TLSMethod

OVERSAMPLE = 10                     # phase bins per shortest box (bins_per_duration)
# the segmentation of period grids (the settings' defaults)
FACTOR, MIN_FRAC, MAX_FRAC, MIN_DAYS = 2.0, 0.01, 0.12, 0.01
SHORT_PERIODS = (0.3, 13.0)         # 27 d curves
LONG_PERIODS = (0.5, 400.0)         # four-year curves
ROW_FIELDS = ("period", "power", "depth", "depth_snr", "duration", "t0", "sde")
N_BEST = 10                         # peaks per result row


# ---- the cases -------------------------------------------------------------------

def listed():
    return [
        # the smallest call: an interactive look at a short curve on a coarse grid
        dict(name="quick_look", kind="power", points=300, periods=1000, durations=3,
             span=30.0, p_lo=0.5, p_hi=10.0, objective="snr", errors="none"),
        # one curve at a time through the kernel-level entry, likelihood objective
        dict(name="single_curve", kind="power", points=2000, periods=10000, durations=5,
             span=90.0, p_lo=0.5, p_hi=30.0, objective="likelihood", errors="unit"),
        # one ground-based survey star over years, per-point errors, its default
        # grid between 0.5 and 4 days, the spectrum back as a periodogram
        dict(name="survey_star", kind="star", points=900, span=2175.0, p_lo=0.5, p_hi=4.0,
             errors="typical"),
        # the batched search: 27 d curves of every length, one weight per curve,
        # one shared grid, result rows back
        dict(name="batch_rows", kind="rows", curves=96, periods=50000, errors="none"),
        # the same curves with per-point photometric errors, whole spectra back
        dict(name="batch_errors", kind="spectra", curves=16, periods=50000, errors="typical"),
        # errors with a heavy tail (clouds, saturation): weights over many decades
        dict(name="batch_outliers", kind="spectra", curves=8, periods=50000, errors="outliers"),
        # four-year curves of 60,000 points over 200,000 periods and 12 box widths
        dict(name="long_baseline", kind="long", curves=4, periods=200000, durations=12),
        # a catalogue: every curve with its own length, baseline and default grid
        dict(name="catalogue_rows", kind="catalogue", curves=1024),
        # one star in six bands, one box shared by the bands
        dict(name="shared_box_star", kind="shared", points=2000, bands=6, span=90.0),
        # transit least squares of Kepler-like curves on the default grid
        dict(name="transit_curves", kind="tls", curves=3, points=20000, p_lo=0.5, p_hi=12.0),
        # the proposal network on one chunk of curves
        dict(name="network_chunk", kind="infer", batch=1024),
        # one training step of the network from its committed weights: logits, loss
        # and every gradient
        dict(name="network_step", kind="train", batch=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    limit = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(("power", "star", "rows", "spectra", "long", "catalogue", "shared",
                           "tls", "infer", "train"))
        if kind == "power":
            case = dict(points=_log_int(rng, 100, 5000), periods=_log_int(rng, 500, 20000),
                        durations=rng.randint(1, 8), span=round(rng.uniform(20.0, 200.0), 3),
                        p_lo=round(rng.uniform(0.4, 1.0), 3), p_hi=round(rng.uniform(5.0, 30.0), 3),
                        objective=rng.choice(("snr", "likelihood")),
                        errors=rng.choice(("none", "unit", "typical", "outliers")))
        elif kind == "star":
            case = dict(points=_log_int(rng, 100, 5000), span=round(rng.uniform(300.0, 2500.0), 3),
                        p_lo=round(rng.uniform(0.4, 1.0), 3), p_hi=round(rng.uniform(2.0, 8.0), 3),
                        errors=rng.choice(("none", "typical", "outliers")))
        elif kind == "rows":
            case = dict(curves=_log_int(rng, 8, 96), periods=_log_int(rng, 5000, 50000),
                        errors=rng.choice(("none", "typical")))
        elif kind == "spectra":
            case = dict(curves=_log_int(rng, 2, 16), periods=_log_int(rng, 5000, 50000),
                        errors=rng.choice(("none", "typical", "outliers")))
        elif kind == "long":
            case = dict(curves=rng.randint(1, 4), periods=_log_int(rng, 20000, 200000),
                        durations=rng.randint(6, 12))
        elif kind == "catalogue":
            case = dict(curves=_log_int(rng, 32, 1024))
        elif kind == "shared":
            case = dict(points=_log_int(rng, 600, 3000), bands=rng.randint(3, 6),
                        span=round(rng.uniform(40.0, 120.0), 3))
        elif kind == "tls":
            case = dict(curves=rng.randint(1, 3), points=_log_int(rng, 2000, 29000),
                        p_lo=round(rng.uniform(0.5, 2.0), 3), p_hi=round(rng.uniform(6.0, 12.0), 3))
        elif kind == "infer":
            case = dict(batch=_log_int(rng, 1, 1024))
        else:
            case = dict(batch=8 * rng.randint(2, 32))
        case["kind"] = kind
        if work(case)["flops"] <= limit:
            return case


# ---- inputs -----------------------------------------------------------------------

def _errors(rng, n, sigma, errors):
    if errors == "none":
        return None
    if errors == "unit":
        return np.ones(n)
    dy = sigma * rng.uniform(0.7, 1.4, n)
    if errors == "outliers":
        bad = rng.random(n) < 0.03
        dy[bad] *= 10.0 ** rng.uniform(0.7, 2.0, int(bad.sum()))
        dy[int(rng.integers(n))] = 60.0 * sigma     # one at least: never a narrow range
    return dy


def _survey_curve(seed, n, span, errors):
    """Irregular sampling over ``span`` days, 1e-3 noise, a 4e-3 transit."""
    rng = np.random.default_rng(seed)
    t = np.sort(rng.uniform(0.0, span, n))
    t[0], t[-1] = 0.0, span
    sigma = 1e-3
    dy = _errors(rng, n, sigma, errors)
    noise = dy if errors in ("typical", "outliers") else sigma
    y = 1.0 + rng.normal(0.0, 1.0, n) * noise
    period = rng.uniform(1.0, 4.0)
    y[np.mod(t - rng.uniform(0.0, period), period) < 0.1] -= 4e-3
    return t + 2458000.0, y, dy


def _batch_curves(case, seed):
    """The batched workload's curves (synthetic.batched_curves) as (t, y, dy)."""
    out = []
    for i, c in enumerate(synthetic.batched_curves(case["curves"], seed=seed)):
        rng = np.random.default_rng([seed, i, 1])
        sigma = float(np.std(np.diff(c.y))) / math.sqrt(2.0)
        out.append((c.t, c.y, _errors(rng, c.t.size, sigma, case["errors"])))
    return out


def _catalogue_curves(case, seed):
    """Curves of 500-6,000 points, every one with its own baseline of 10-27 d."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(case["curves"]):
        n = int(rng.integers(500, 6001))
        t = np.sort(rng.uniform(0.0, rng.uniform(10.0, 27.0), n)) + 2460000.0
        sigma = 10.0 ** rng.uniform(np.log10(2e-4), np.log10(5e-3))
        y = 1.0 + rng.normal(0.0, sigma, n)
        if rng.random() < 0.5:
            period = rng.uniform(0.5, 8.0)
            y[np.mod(t, period) < rng.uniform(0.02, 0.25)] -= 10.0 ** rng.uniform(-4.0, -2.0)
        out.append((t, y.astype(np.float32).astype(np.float64), None))
    return out


def _band_curves(case, seed):
    span, total = case["span"], case["points"]
    star = synthetic.multiband_stars(1, seed=seed, span=span, n_range=(total, total))[0]
    names = list(star)[-case["bands"]:]
    # every star of a field has the survey's first and last night
    star[names[-1]].t[[0, -1]] = 2460000.05, 2460000.05 + span - 0.55
    return {b: star[b] for b in names}


def _tls_curves(case, seed):
    return synthetic.tls_curves(case["curves"], seed=seed,
                                n_range=(case["points"], int(case["points"] * 1.03)))


def _net_inputs(case, seed):
    """Binned curves: standardised bin means and an occupancy flag, bf16."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["batch"], N_BINS)
    occ = (torch.rand(shape, generator=g, device="cuda") < 0.85).float()
    mean = torch.randn(shape, generator=g, device="cuda") * 0.6 * occ
    x = torch.stack([mean, occ], dim=2).to(torch.bfloat16).contiguous()
    # a curve's best period lies among the grid's long ones far more often than not
    labels = torch.randint(3 * N_CLASSES // 4, N_CLASSES, (case["batch"],), dtype=torch.int32, generator=g,
                           device="cuda")
    return x, labels


def _weights():
    return Weights.load(os.path.join(os.path.dirname(cuperiod_b200.__file__),
                                     "proposal_weights.npz"))


# ---- period grids (plain numpy) ------------------------------------------------------

def _durations(p_lo, n):
    hi = MAX_FRAC * p_lo
    lo = max(MIN_FRAC * p_lo, MIN_DAYS)
    return np.array([hi]) if lo >= hi else np.geomspace(lo, hi, n)


def _log_segments(periods, n_dur):
    """A period grid's ``(periods, durations)`` segments, a factor of two each."""
    p0 = float(periods.min())
    index = np.floor(np.log(periods / p0) / math.log(FACTOR) + 1e-9).astype(np.int64)
    return [(np.ascontiguousarray(periods[index == k]), _durations(p0 * FACTOR ** k, n_dur))
            for k in np.unique(index).tolist()]


def _default_segments(baseline, p_lo, p_hi, oversample, n_dur=8, frac=0.05):
    """The default grid: per segment uniform in frequency, the step a fraction of
    the baseline's resolution."""
    top = min(p_hi, baseline / 2.0)
    df = frac / (oversample * baseline)
    out = []
    lo = p_lo
    while lo < top:
        hi = min(lo * FACTOR, top)
        f = np.arange(1.0 / hi, 1.0 / lo, df)
        f = f[f < 1.0 / lo]
        if f.size:
            out.append((1.0 / f[::-1], _durations(lo, n_dur)))
        lo = hi
    return out


def _segments(case):
    """The trial segments of a case whose grid does not depend on its curves."""
    kind = case["kind"]
    if kind == "power":
        periods = np.geomspace(case["p_lo"], case["p_hi"], case["periods"])
        return [(periods, 0.05 + 0.03 * np.arange(case["durations"]))]
    if kind == "star":
        t = _survey_curve(0, case["points"], case["span"], "none")[0]
        return _default_segments(float(t.max() - t.min()), case["p_lo"], case["p_hi"], 1)
    if kind in ("rows", "spectra"):
        return _log_segments(np.geomspace(*SHORT_PERIODS, case["periods"]), 8)
    if kind == "long":
        return _log_segments(np.geomspace(*LONG_PERIODS, case["periods"]), case["durations"])
    if kind == "catalogue":
        return _default_segments(18.5, 0.2, 100.0, 2)      # the mean baseline's
    if kind == "shared":
        return _default_segments(case["span"] - 0.55, 0.2, 100.0, 2)
    raise ValueError(kind)


def _bins(periods, durations):
    """Bin width, box widths in bins and phase bins per period (with the pad)."""
    bin_ = float(durations.min()) / OVERSAMPLE
    widths = []
    for d in durations.tolist():
        k = math.floor(d / bin_ + 0.5)
        if k >= 1 and k not in widths:
            widths.append(k)
    width = int(math.ceil(float(periods.max()) / bin_)) + OVERSAMPLE + 1
    nb = np.minimum(np.ceil(periods / bin_).astype(np.int64) + OVERSAMPLE, width - 1)
    return bin_, widths, width, nb


def _tls_periods(case):
    baseline = 29999 * (30.0 / 1440.0)
    top = min(case["p_hi"], baseline / 2.0)
    df = 0.02 / (2 * baseline)
    return 1.0 / np.arange(1.0 / top, 1.0 / case["p_lo"], df)[::-1]


# ---- prepare and run -------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "power":
        state["curve"] = _survey_curve(seed, case["points"], case["span"], case["errors"])
        state["periods"], state["durations"] = _segments(case)[0]
    elif kind == "star":
        t, y, dy = _survey_curve(seed, case["points"], case["span"], case["errors"])
        state["curve"] = LightCurve(t, y, dy, Domain.FLUX)
        state["settings"] = BLSSettings(min_period_days=case["p_lo"],
                                        max_period_days=case["p_hi"], grid_oversample=1)
    elif kind in ("rows", "long"):
        if kind == "rows":
            curves = _batch_curves(case, seed)
            edges, n_dur = SHORT_PERIODS, 8
        else:
            curves = [(c.t, c.y, None)
                      for c in synthetic.long_baseline_curves(case["curves"], seed=seed)]
            edges, n_dur = LONG_PERIODS, case["durations"]
        state["curves"] = [(f"c{i}", LightCurve(*c, Domain.FLUX)) for i, c in enumerate(curves)]
        state["grid"] = GridSpec(kind="period", values=np.geomspace(*edges, case["periods"]))
        state["settings"] = BLSSettings(n_durations=n_dur)
    elif kind == "spectra":
        state["curves"] = _batch_curves(case, seed)
        state["segments"] = _segments(case)
    elif kind == "catalogue":
        state["curves"] = [(f"c{i}", LightCurve(*c, Domain.FLUX))
                           for i, c in enumerate(_catalogue_curves(case, seed))]
        state["settings"] = BLSSettings()
    elif kind == "shared":
        state["star"] = MultiBandLightCurve.from_light_curves(
            {b: LightCurve(c.t, c.y, c.dy, Domain.FLUX)
             for b, c in _band_curves(case, seed).items()})
        state["settings"] = BLSSettings(mb_ephemeris="shared")
        state["grid"] = multiband_default_grid(BLSMethod(), state["star"], state["settings"])
    elif kind == "tls":
        state["curves"] = [LightCurve(c.t, c.y, c.dy, Domain.FLUX) for c in _tls_curves(case, seed)]
        state["settings"] = TLSSettings(min_period_days=case["p_lo"],
                                        max_period_days=case["p_hi"])
        state["method"] = TLSMethod()
        state["grid"] = state["method"].default_grid(state["curves"][0], state["settings"])
    else:
        state["x"], state["labels"] = _net_inputs(case, seed)
        state["net"] = ProposalNet(_weights(), train=kind == "train")
    return state


def _columns(rows):
    """Result rows as arrays: what a table of them holds."""
    nan = math.nan
    out = {k: np.array([[r.get(f"{k}_{i}", nan) for i in range(1, N_BEST + 1)] for r in rows])
           for k in ROW_FIELDS}
    for k in ("best_period", "n_samples", "baseline"):
        out[k] = np.array([r[k] for r in rows])
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "power":
        t, y, dy = state["curve"]
        p = bls_power(t, y, np.ones_like(t) if dy is None else dy, state["periods"],
                      state["durations"], OVERSAMPLE, objective=case["objective"])
        return (p.power, p.depth, p.depth_err, p.depth_snr, p.duration, p.transit_time,
                p.log_likelihood)
    if kind == "star":
        pg = periodogram(state["curve"], "BLS", settings=state["settings"])
        return (pg.frequency, pg.power, *(pg.extras[k] for k in ("depth", "depth_snr", "duration",
                                                                 "t0", "sde")))
    if kind in ("rows", "long"):
        done = batch_periodograms(state["curves"], "BLS", grid=state["grid"],
                                  settings=state["settings"])
        return _columns(done.rows)
    if kind == "spectra":
        return bls_power_many(state["curves"], state["segments"], OVERSAMPLE)
    if kind == "catalogue":
        return _columns(batch_periodograms(state["curves"], "BLS",
                                           settings=state["settings"]).rows)
    if kind == "shared":
        pg = bls_multiband_power(state["grid"], state["star"], state["settings"])
        return (pg.power, *(pg.extras[k] for k in ("depth", "depth_snr", "duration", "t0", "sde",
                                                   "band_index")))
    if kind == "tls":
        pgs = state["method"].power_many(state["grid"], state["curves"], state["settings"])
        return [(pg.power, *(pg.extras[k] for k in ("sr", "depth", "duration", "t0")))
                for pg in pgs]
    net = state["net"]
    logits = net.forward(state["x"])
    if kind == "infer":
        return logits
    dlogits, loss = net.loss_and_grad(logits, state["labels"])
    net.zero_grad()
    net.backward(dlogits)
    return {"logits": logits, "loss": loss, "gradients": list(net.g)}


# ---- the least work of one pass -----------------------------------------------------------

def _search_work(segments, points, curves, fields):
    """``points``: of all curves together.  A fold is a product, a floor, a
    scaling and the sums; a box two differences, two quotients and a bound."""
    n_periods = sum(p.size for p, _ in segments)
    boxes = 0.0
    for p, d in segments:
        _, widths, _, nb = _bins(p, d)
        boxes += sum(float(np.maximum(nb - w + 1, 0).sum()) for w in widths)
    return n_periods, 6.0 * points * n_periods + 10.0 * curves * boxes


def work(case):
    kind = case["kind"]
    if kind in ("power", "star"):
        segments = _segments(case)
        n_per, flops = _search_work(segments, case["points"], 1, 7)
        return {"bytes": 24.0 * case["points"] + 8.0 * n_per * 8, "flops": flops}
    if kind in ("rows", "spectra", "long", "catalogue"):
        mean = {"rows": 9900.0, "spectra": 9900.0, "long": 60000.0, "catalogue": 3250.0}[kind]
        n = mean * case["curves"]
        n_per, flops = _search_work(_segments(case), n, case["curves"], 7)
        out = 7.0 * 8 * n_per * case["curves"] if kind == "spectra" else 640.0 * case["curves"]
        per_point = 16.0 if case.get("errors", "none") == "none" else 24.0
        return {"bytes": per_point * n + 8.0 * n_per + out, "flops": flops}
    if kind == "shared":
        n_per, flops = _search_work(_segments(case), case["points"], case["bands"], 7)
        return {"bytes": 24.0 * case["points"] + 8.0 * n_per * 7, "flops": flops}
    if kind == "tls":
        n_per = _tls_periods(case).size
        per_curve = 6.0 * case["points"] + 256 * 8.0 * sum(_tls_widths())
        return {"bytes": case["curves"] * (24.0 * case["points"] + 40.0 * n_per),
                "flops": case["curves"] * n_per * per_curve}
    b, length, macs, weights = case["batch"], N_BINS, 0.0, 0
    c = IN_CHANNELS
    for _ in range(N_CONV):
        length //= 2
        macs += float(length) * CHANNELS * WIDTH * c
        weights += CHANNELS * WIDTH * c
        c = CHANNELS
    flat = CHANNELS * length
    macs += flat * HIDDEN + HIDDEN * N_CLASSES
    weights += flat * HIDDEN + HIDDEN * N_CLASSES
    io = b * (N_BINS * IN_CHANNELS * 2.0 + N_CLASSES * 4.0)
    if kind == "infer":
        return {"bytes": io + 2.0 * weights, "flops": 2.0 * b * macs}
    # the backward pass: one product for the weights, one for the inputs of every
    # layer but the first
    first = float(N_BINS // 2) * CHANNELS * WIDTH * IN_CHANNELS
    return {"bytes": io + 2.0 * weights + 4.0 * weights,
            "flops": 2.0 * b * (3.0 * macs - first)}


# ---- what a pass returns, in 64 bits ---------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_device())


def _fold(tau, values, periods, bin_, width):
    """Per period the bin sums of every column of ``values``: (K, periods, width)."""
    w = tau[None, :] - periods[:, None] * torch.floor(tau[None, :] / periods[:, None])
    ind = ((w / bin_).to(torch.int64) + 1).clamp_(0, width - 1)
    out = []
    for v in values:
        h = torch.zeros((periods.numel(), width), dtype=torch.float64, device=tau.device)
        out.append(h.scatter_add_(1, ind, v[None, :].expand(periods.numel(), -1)))
    return out


def _pad(h, nb):
    """The first bins repeated over the last ones, per period."""
    rows = torch.arange(h.shape[0], device=h.device)
    for k in range(OVERSAMPLE):
        dst = nb - OVERSAMPLE + k
        ok = (dst >= 0) & (dst < h.shape[1])
        h[rows[ok], dst[ok]] = h[rows[ok], 1 + k]
    return torch.cumsum(h, dim=1)


def _box_terms(cy, ci, d, sum_y, sum_i, floor):
    """Depth and inside/outside weights of every box of width ``d``, with whether
    the box is admissible and a dip."""
    y_in, i_in = cy[:, d:] - cy[:, :-d], ci[:, d:] - ci[:, :-d]
    i_out = sum_i - i_in
    ok = (i_in >= floor) & (i_out >= floor)
    one = torch.ones_like(i_in)
    a, b = torch.where(ok, i_in, one), torch.where(ok, i_out, one)
    depth = (sum_y - y_in) / b - y_in / a
    return depth, a, b, ok & (depth >= 0.0)


def _objective(depth, a, b, objective):
    if objective == "snr":
        return depth / torch.sqrt(1.0 / a + 1.0 / b)
    return 0.5 * a * depth * depth


def _bls_exact(t, y, dy, segments, objective="snr"):
    """The seven fields of every trial period of one curve: (7, periods)."""
    t_min = float(t.min())
    tau = _dev(t - t_min)
    iv = np.ones(t.size) if dy is None else 1.0 / (dy * dy)
    yw = (y - np.median(y)) * iv
    sum_y, sum_i = float(yw.sum()), float(iv.sum())
    floor = 4.0 * t.size * float(np.finfo(np.float64).eps) * sum_i
    values = (_dev(yw), _dev(iv))
    out = []
    for periods, durations in segments:
        bin_, widths, width, nb_all = _bins(periods, durations)
        step = max(1, min(periods.size, 40_000_000 // max(t.size, width)))
        for lo in range(0, periods.size, step):
            p = _dev(periods[lo:lo + step])
            nb = _dev(nb_all[lo:lo + step])
            hy, hi = _fold(tau, values, p, bin_, width)
            cy, ci = _pad(hy, nb), _pad(hi, nb)
            best = torch.full((p.numel(),), -math.inf, dtype=torch.float64, device=p.device)
            bn, bd = torch.zeros_like(nb), torch.zeros_like(nb)
            for d in widths:
                if d >= width:
                    continue
                depth, a, b, ok = _box_terms(cy, ci, d, sum_y, sum_i, floor)
                start = torch.arange(depth.shape[1], device=p.device)
                ok &= (start[None, :] + d <= nb[:, None]) & (d < nb[:, None])
                v = torch.where(ok, _objective(depth, a, b, objective),
                                torch.full_like(depth, -math.inf))
                top = v.max(dim=1).values
                n = (v == top[:, None]).to(torch.int8).argmax(dim=1)     # the first of equals
                better = top > best
                best, bn = torch.where(better, top, best), torch.where(better, n, bn)
                bd = torch.where(better, torch.full_like(bd, d), bd)
            rows = torch.arange(p.numel(), device=p.device)
            y_in = cy[rows, bn + bd] - cy[rows, bn]
            i_in = ci[rows, bn + bd] - ci[rows, bn]
            found = torch.isfinite(best)
            a = torch.where(found, i_in, torch.ones_like(i_in))
            b = torch.where(found, sum_i - i_in, torch.ones_like(i_in))
            depth = (sum_y - y_in) / b - y_in / a
            err = torch.sqrt(1.0 / a + 1.0 / b)
            dur = bd.double() * bin_
            t0 = torch.fmod(bn.double() * bin_ + 0.5 * dur, p) + t_min
            fields = torch.stack([depth, err, depth / err, dur, t0, 0.5 * a * depth * depth])
            fields = torch.where(found[None, :], fields, torch.zeros_like(fields))
            out.append(torch.cat([best[None, :], fields]).cpu().numpy())
    return np.concatenate(out, axis=1)


def _sde(power):
    std = float(power.std())
    return (power - float(power.mean())) / std if std > 0.0 else np.zeros_like(power)


def _shared_exact(bands, segments):
    """Power, depth, depth SNR, duration, epoch and band of the shared box."""
    t_min = min(float(c.t.min()) for c in bands)
    info = []
    for c in bands:
        iv = 1.0 / (c.dy * c.dy)
        yw = (c.y - np.median(c.y)) * iv
        si = float(iv.sum())
        info.append((_dev(c.t - t_min), (_dev(yw), _dev(iv)), float(yw.sum()), si,
                     4.0 * c.t.size * float(np.finfo(np.float64).eps) * si))
    out = []
    for periods, durations in segments:
        bin_, widths, width, nb_all = _bins(periods, durations)
        step = max(1, min(periods.size, 20_000_000 // width))
        for lo in range(0, periods.size, step):
            p, nb = _dev(periods[lo:lo + step]), _dev(nb_all[lo:lo + step])
            sums = []
            for tau, values, *_ in info:
                hy, hi = _fold(tau, values, p, bin_, width)
                sums.append((_pad(hy, nb), _pad(hi, nb)))
            best = torch.full((p.numel(),), -math.inf, dtype=torch.float64, device=p.device)
            bn, bd = torch.zeros_like(nb), torch.zeros_like(nb)
            for d in widths:
                if d >= width:
                    continue
                total, hit = 0.0, False
                for (cy, ci), (_, _, sy, si, floor) in zip(sums, info):
                    depth, a, b, ok = _box_terms(cy, ci, d, sy, si, floor)
                    total = total + torch.where(ok, depth * depth / (1.0 / a + 1.0 / b),
                                                torch.zeros_like(depth))
                    hit = hit | ok
                start = torch.arange(total.shape[1], device=p.device)
                hit &= (start[None, :] + d <= nb[:, None]) & (d < nb[:, None])
                v = torch.where(hit, total, torch.full_like(total, -math.inf))
                top = v.max(dim=1).values
                n = (v == top[:, None]).to(torch.int8).argmax(dim=1)
                better = top > best
                best, bn = torch.where(better, top, best), torch.where(better, n, bn)
                bd = torch.where(better, torch.full_like(bd, d), bd)
            rows = torch.arange(p.numel(), device=p.device)
            depths, snrs = [], []
            for (cy, ci), (_, _, sy, si, floor) in zip(sums, info):
                y_in = cy[rows, bn + bd] - cy[rows, bn]
                i_in = ci[rows, bn + bd] - ci[rows, bn]
                ok = (i_in >= floor) & (si - i_in >= floor)
                a = torch.where(ok, i_in, torch.ones_like(i_in))
                b = torch.where(ok, si - i_in, torch.ones_like(i_in))
                depth = (sy - y_in) / b - y_in / a
                ok &= depth >= 0.0
                zero = torch.zeros_like(depth)
                depths.append(torch.where(ok, depth, zero))
                snrs.append(torch.where(ok, depth / torch.sqrt(1.0 / a + 1.0 / b), zero))
            snr = torch.stack(snrs)
            band = snr.argmax(dim=0)
            power = (snr * snr).sum(dim=0)
            depth = torch.stack(depths).gather(0, band[None, :])[0]
            dur = bd.double() * bin_
            t0 = torch.fmod(bn.double() * bin_ + 0.5 * dur, p) + t_min
            fields = torch.stack([power, depth, torch.sqrt(power), dur, t0, band.double()])
            found = torch.isfinite(best)
            out.append(torch.where(found[None, :], fields, torch.zeros_like(fields)).cpu().numpy())
    return np.concatenate(out, axis=1)


def _tls_widths(n_bins=256):
    fracs = np.geomspace(0.01, 0.10, 5)
    return sorted({min(max(int(round(f * n_bins)), 1), n_bins - 1) for f in fracs})


def _tls_template(n, u1=0.4, u2=0.3):
    if n <= 1:
        return np.ones(max(n, 1))
    x = (np.arange(n) + 0.5) / n - 0.5
    mu = np.sqrt(1.0 - np.clip(2.0 * np.abs(x), 0.0, 1.0) ** 2)
    g = 1.0 - u1 * (1.0 - mu) - u2 * (1.0 - mu) ** 2
    g = np.where(2.0 * np.abs(x) < 1.0, g, 0.0)
    return g / g.max()


def _tls_exact(curve, periods, n_bins=256):
    """SDE, signal residue, depth, duration and epoch per trial period."""
    t, y, dy = curve.t, curve.y, curve.dy
    t_ref = float(t.min())
    scale = 2.0 ** round(math.log2(float(np.median(np.abs(dy)))))
    w = 1.0 / (dy / scale) ** 2
    total = float(w.sum())
    yw = w * (y / scale - float((w * (y / scale)).sum()) / total)
    tau, values = _dev(t - t_ref), (_dev(yw), _dev(w))
    widths = _tls_widths(n_bins)
    out = []
    step = max(1, 40_000_000 // t.size)
    for lo in range(0, periods.size, step):
        p = _dev(periods[lo:lo + step])
        q = tau[None, :] / p[:, None]
        ind = ((q - torch.floor(q)) * n_bins).to(torch.int64).clamp_(0, n_bins - 1)
        a, b = (torch.zeros((p.numel(), n_bins), dtype=torch.float64, device=p.device)
                .scatter_add_(1, ind, v[None, :].expand(p.numel(), -1)) for v in values)
        a, b = (torch.cat([h, h[:, :max(widths) - 1]], dim=1) for h in (a, b))
        best = torch.zeros(p.numel(), dtype=torch.float64, device=p.device)
        depth, dur, t0 = torch.zeros_like(best), torch.zeros_like(best), torch.zeros_like(best)
        rows = torch.arange(p.numel(), device=p.device)
        for wd in widths:
            g = _tls_template(wd)
            num = sum(float(g[k]) * a[:, k:k + n_bins] for k in range(wd))
            cwg = sum(float(g[k]) * b[:, k:k + n_bins] for k in range(wd))
            den = sum(float(g[k]) * float(g[k]) * b[:, k:k + n_bins] for k in range(wd))
            de = den - cwg * cwg / total
            ok = (num < 0.0) & (den > 1e-300) & (de > 1e-9 * den)
            safe = torch.where(ok, de, torch.ones_like(de))
            sr = torch.where(ok, num * num / safe, torch.zeros_like(de))
            top = sr.max(dim=1).values
            s = (sr == top[:, None]).to(torch.int8).argmax(dim=1)
            better = top > best
            centre = (s.double() + wd / 2.0) / n_bins
            best = torch.where(better, top, best)
            depth = torch.where(better, -num[rows, s] / safe[rows, s], depth)
            dur = torch.where(better, wd / n_bins * p, dur)
            t0 = torch.where(better, (centre - torch.floor(centre)) * p, t0)
        out.append(torch.stack([best, depth * scale, dur, t0 + t_ref]).cpu().numpy())
    sr, depth, dur, t0 = np.concatenate(out, axis=1)
    return tuple(v[::-1].copy() for v in (_sde(sr), sr, depth, dur, t0))


def _net_exact(case, seed):
    x, labels = _net_inputs(case, seed)
    params = [torch.tensor(a, device="cuda") for a in _weights().arrays()]
    # the matrices as the network multiplies them (bf16), the biases as they are
    params = [(a.to(torch.bfloat16) if a.ndim == 2 else a).double().requires_grad_(True)
              for a in params]

    def forward(x):
        act = x.double().permute(0, 2, 1)
        for layer in range(N_CONV):
            c = IN_CHANNELS if layer == 0 else CHANNELS
            w = params[layer][:, :WIDTH * c].reshape(CHANNELS, WIDTH, c).permute(0, 2, 1)
            act = torch.relu(torch.nn.functional.conv1d(act, w, params[N_CONV + layer], stride=2,
                                                        padding=3))
        flat = act.permute(0, 2, 1).reshape(act.shape[0], -1)
        h = torch.relu(flat @ params[2 * N_CONV].T + params[2 * N_CONV + 1])
        return h @ params[2 * N_CONV + 2].T + params[2 * N_CONV + 3]

    n = x.shape[0]
    if case["kind"] == "infer":
        with torch.no_grad():
            return torch.cat([forward(x[i:i + 64]) for i in range(0, n, 64)])
    target = torch.zeros((n, N_CLASSES), dtype=torch.float64, device="cuda")
    lab, rows = labels.long(), torch.arange(n, device="cuda")
    target[rows, lab] += 0.8
    target[rows, (lab - 1).clamp_min(0)] += 0.1
    target[rows, (lab + 1).clamp_max(N_CLASSES - 1)] += 0.1
    logits, loss = [], 0.0
    for i in range(0, n, 64):
        z = forward(x[i:i + 64])
        part = -(target[i:i + 64] * torch.log_softmax(z, dim=1)).sum()
        (part / n).backward()
        logits.append(z.detach())
        loss = loss + part.detach()
    return {"logits": torch.cat(logits), "loss": loss.reshape(1),
            "gradients": [p.grad for p in params]}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("infer", "train"):
        return _net_exact(case, seed)
    if kind == "power":
        t, y, dy = _survey_curve(seed, case["points"], case["span"], case["errors"])
        return tuple(_bls_exact(t, y, dy, _segments(case), case["objective"]))
    if kind == "star":
        t, y, dy = _survey_curve(seed, case["points"], case["span"], case["errors"])
        segments = _segments(case)
        f = _bls_exact(t, y, dy, segments)
        period = np.concatenate([p for p, _ in segments])
        power = np.nan_to_num(f[0], nan=0.0, posinf=0.0, neginf=0.0)
        return tuple(v[::-1].copy() for v in (1.0 / period, power, f[1], f[3], f[4], f[5],
                                              _sde(power)))
    if kind == "spectra":
        return np.stack([_bls_exact(t, y, dy, _segments(case))
                         for t, y, dy in _batch_curves(case, seed)], axis=1)
    if kind == "shared":
        bands = list(_band_curves(case, seed).values())
        times = np.concatenate([c.t for c in bands])
        segments = _default_segments(float(times.max() - times.min()), 0.2, 100.0, 2)
        power, depth, snr, dur, t0, band = _shared_exact(bands, segments)
        return tuple(v[::-1].copy() for v in (power, depth, snr, dur, t0, _sde(power), band))
    if kind == "tls":
        curves = _tls_curves(case, seed)
        span = float(curves[0].t.max() - curves[0].t.min())
        top = min(case["p_hi"], span / 2.0)
        periods = 1.0 / np.arange(1.0 / top, 1.0 / case["p_lo"], 0.02 / (2 * span))[::-1]
        return [_tls_exact(c, periods) for c in curves]
    # whole batches searched and ranked: a minute and more in plain torch
    return None
