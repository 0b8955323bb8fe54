"""The search kernel's histogram encodings and scan shapes at the sizes where they
change, against the oracle.

Encodings: one weight with at most 4,000 points in any phase bin (two words) or more
(three words); per-point weights in 38-bit (at most 8,191 points in a bin) or 61-bit
fixed point.  The search sums quantised values exactly, at worst 2^-24 of the largest
per point with one weight, so a power agrees within 1e-6; the boxes are the reference's
except where rounding decides between near ties.
"""

from __future__ import annotations

import numpy as np
import pytest

from _cases import FIELDS, compare, transit_curve
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    from cuperiod_b200 import _lib
    eng = _lib.Engine()
    yield eng
    eng.close()


def _check(engine, t, y, dy, periods, durations, objective="snr"):
    from cuperiod_b200.core import bls_power
    ref = oracle.bls_power(t, y, dy, periods, durations, 10, objective=objective)
    out = bls_power(t, y, dy, periods, durations, 10, objective=objective, engine=engine)
    got = {f: getattr(out, f) for f in FIELDS}
    # adjacent periods of these short grids share their best box, so their powers tie to
    # the last bits and the best of them is not compared
    compare(ref, got, rtol=1e-6, box_agree=0.98)


def _errors(rng, n, weights):
    return {"one": np.full(n, 1e-3), "narrow": 1e-3 * rng.uniform(0.7, 1.4, n),
            "spread": 1e-3 * 10.0 ** rng.uniform(0.0, 2.5, n)}[weights]


def _bursts(n, per_burst, seed):
    """Bursts of points within seconds, one a day at the same time of day: a period of
    a day folds all of them into one bin."""
    rng = np.random.default_rng(seed)
    t = np.floor(np.arange(n) / per_burst) + 0.3 + np.sort(rng.uniform(0.0, 5e-4, n)) % 5e-4
    t = np.sort(t)
    y = 1.0 + rng.normal(0.0, 1e-3, n)
    y[np.mod(t, 3.7) < 0.2] -= 4e-3
    return t, y, rng


@pytest.mark.parametrize("objective", ["snr", "likelihood"])
@pytest.mark.parametrize("weights", ["one", "narrow", "spread"])
@pytest.mark.parametrize("n,per_burst", [(4000, 200), (4001, 200), (9000, 450), (9000, 9000 // 8)])
def test_many_points_in_one_bin(engine, n, per_burst, weights, objective):
    t, y, rng = _bursts(n, per_burst, n)
    t[: n // 4] += np.sort(rng.uniform(0.0, 0.9, n // 4))      # some spread, for other boxes
    t = np.sort(t)
    periods = np.concatenate([np.linspace(0.9, 1.1, 41), np.linspace(1.9, 2.1, 21)])
    _check(engine, t, y, _errors(rng, n, weights), periods, np.array([0.05, 0.08, 0.12]),
           objective)


@pytest.mark.parametrize("weights", ["one", "narrow", "spread"])
@pytest.mark.parametrize("n", [5, 255, 256, 257, 511, 513, 1023, 1025, 2047, 2048, 2049, 4097, 6200])
def test_point_counts_around_the_chunks(engine, n, weights):
    rng = np.random.default_rng(n)
    t, y, _ = transit_curve(n, span=30.0, period=2.1, depth=6e-3, duration=0.2, seed=n)
    periods = np.geomspace(0.6, 6.0, 150)
    if n < 20:
        periods = periods[:20]
    dy = _errors(rng, n, weights)
    from cuperiod_b200.core import bls_power
    ref = oracle.bls_power(t, y, dy, periods, np.array([0.05, 0.1, 0.2]), 10)
    out = bls_power(t, y, dy, periods, np.array([0.05, 0.1, 0.2]), 10, engine=engine)
    # a handful of points ties its boxes: only the power is compared there
    compare(ref, {f: getattr(out, f) for f in FIELDS}, rtol=1e-6,
            box_agree=0.0 if n < 20 else 0.98)


@pytest.mark.parametrize("weights", ["one", "narrow", "spread"])
@pytest.mark.parametrize("bins", [9, 10, 11, 31, 245, 246, 247, 503, 1270, 2292, 2293, 2294, 2600,
                                  4700, 5200])
def test_bin_counts_around_the_scan_blocks(engine, bins, weights):
    # `bins` phase bins plus the 10 of the pad: the pad overlapping its source (few
    # bins), each lane's run of bins, and more bins than one scan block holds
    rng = np.random.default_rng(bins)
    n = 1500
    t, y, _ = transit_curve(n, span=40.0, period=5.0, depth=5e-3, duration=0.5, seed=bins)
    period = 5.0
    bin_ = period / (bins - 0.5)
    durations = np.array([10.0, 14.0, 25.0, 33.0, 60.0])[: 1 if bins < 40 else 5] * bin_
    periods = np.linspace(period * (1 - 2e-3), period * (1 + 0.4 / bins * 0.5), 7)
    _check(engine, t, y, _errors(rng, n, weights), periods, durations)


@pytest.mark.parametrize("weights", ["one", "narrow", "spread"])
@pytest.mark.parametrize("n_dur", [1, 4, 5, 31, 32])
def test_width_counts_around_the_groups(engine, n_dur, weights):
    rng = np.random.default_rng(n_dur)
    t, y, _ = transit_curve(900, span=40.0, period=3.3, depth=5e-3, duration=0.3, seed=n_dur)
    durations = 0.05 + 0.011 * np.arange(n_dur)
    _check(engine, t, y, _errors(rng, 900, weights), np.geomspace(1.0, 5.0, 80), durations)


@pytest.mark.parametrize("weights", ["one", "narrow", "spread"])
def test_sparse_curves_with_tied_boxes(engine, weights):
    # empty bins make boxes tie exactly: the first (duration, start) wins, as in the
    # reference; with per-point weights the reference's own rounding may part them
    rng = np.random.default_rng(3)
    t = np.sort(rng.uniform(0.0, 50.0, 60))
    y = 1.0 + rng.normal(0.0, 1e-3, 60)
    dy = _errors(rng, 60, weights)
    from cuperiod_b200.core import bls_power
    periods, durations = np.geomspace(1.0, 8.0, 300), np.array([0.05, 0.08, 0.12, 0.2])
    ref = oracle.bls_power(t, y, dy, periods, durations, 10)
    out = bls_power(t, y, dy, periods, durations, 10, engine=engine)
    compare(ref, {f: getattr(out, f) for f in FIELDS}, rtol=1e-6,
            box_agree=0.98 if weights == "one" else 0.0)
