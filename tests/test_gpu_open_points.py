"""Points whose phase bin the search's fast fold leaves open, in number: a cadence and
periods that put the points on bin edges (more open points than a tile's list holds), and
more cycles than the fast fold covers (every point of every period), in every encoding,
against the oracle.

The sums are exact or FP64 as elsewhere, so the powers agree within the 1e-6 of the other
search tests; a point in a wrong bin moves a power by far more.  Edges tie boxes, so the
chosen boxes are not compared.
"""

from __future__ import annotations

import numpy as np
import pytest

from _cases import FIELDS, compare
from oracle import oracle

pytestmark = pytest.mark.gpu

WEIGHTS = ["pair", "uniform", "narrow", "spread", "general"]


@pytest.fixture(scope="module")
def engine():
    from cuperiod_b200 import _lib
    eng = _lib.Engine()
    yield eng
    eng.close()


def _check(engine, t, y, weights, periods, durations, fast):
    from cuperiod_b200.core import bls_power
    rng = np.random.default_rng(t.size)
    dy = np.full(t.size, 1e-3)
    if weights == "uniform":            # three words: the curve is not in time order
        t, y = np.roll(t, 7), np.roll(y, 7)
    elif weights == "narrow":
        dy = dy * rng.uniform(0.7, 1.4, t.size)
    elif weights in ("spread", "general"):
        dy = dy * 10.0 ** rng.uniform(0.0, 2.5, t.size)
        if weights == "general":        # FP64 sums: a weight of zero
            dy[t.size // 2] = 1e200
    ref = oracle.bls_power(t, y, dy, periods, durations, 10)
    out = bls_power(t, y, dy, periods, durations, 10, engine=engine)
    assert engine.info()["fast_fold_segments"] == fast
    compare(ref, {f: getattr(out, f) for f in FIELDS}, rtol=1e-6, box_agree=0.0)


def _flux(t, period, seed):
    y = 1.0 + np.random.default_rng(seed).normal(0.0, 1e-3, t.size)
    y[np.mod(t, period) < 0.05 * period] -= 4e-3
    return y


@pytest.mark.parametrize("weights", WEIGHTS)
@pytest.mark.parametrize("n", [300, 1500, 4500, 6200])
def test_points_on_bin_edges(engine, n, weights):
    # the cadence is two bins, the periods are whole bins
    t = np.arange(n) * 0.02
    _check(engine, t, _flux(t, 2.37, n), weights, np.round(np.arange(1.0, 4.0, 0.03), 2),
           np.array([0.1, 0.2, 0.3]), fast=1)


@pytest.mark.parametrize("weights", WEIGHTS)
@pytest.mark.parametrize("n", [4500, 6200])
def test_some_points_on_bin_edges(engine, n, weights):
    # a cadence of a tenth of a bin: edges in the first cycle only
    t = np.arange(n) * 0.001
    _check(engine, t, _flux(t, 1.37, n), weights, np.geomspace(0.4, 2.0, 90),
           np.array([0.1, 0.2]), fast=1)


@pytest.mark.parametrize("weights", WEIGHTS)
@pytest.mark.parametrize("n", [2, 300, 2048, 4500])
def test_more_cycles_than_the_fast_fold_covers(engine, n, weights):
    # ten years of periods of 10 to 20 minutes: up to 530,000 cycles
    t = np.sort(np.random.default_rng(n).uniform(0.0, 3700.0, n))
    t[-1] = 3700.0
    _check(engine, t, _flux(t, 0.0101, n), weights, np.linspace(0.0069, 0.0139, 70),
           np.array([0.0004, 0.0008, 0.0012]), fast=0)
