"""The FP32 screen of curves with per-point weights discards no box that may be the best:
the search equals, bit for bit, the one that evaluates every box in FP64.

Hard for it are curves of which a few points hold nearly all the weight: the weight left
outside a box that holds them, or inside one that does not, is then of the size of FP32's
rounding of the total.  Where those points lie at the start of the curve they fall into the
first phase bins at every period, which the wrap pad repeats, so that the prefix sums end at
up to twice the total.
"""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DURATIONS = np.array([0.05, 0.1, 0.2, 0.3])


def _heavy_start(seed):
    """20 to 120 points over 400 days; one to four at the start, within half the pad of the
    shortest period, weigh 10^4 to 10^7 times the others."""
    rng = np.random.default_rng(seed)
    n = int(rng.integers(20, 121))
    k = int(rng.integers(1, 5))
    heavy = np.sort(rng.uniform(0.0, 0.045, k))
    heavy[0] = 0.0
    t = np.concatenate([heavy, np.sort(rng.uniform(0.06, 400.0, n - k))])
    w = np.full(n, 1.0) * 10 ** rng.uniform(-0.5, 0.5, n)
    w[:k] = 10 ** rng.uniform(4, 7) * rng.uniform(0.5, 1.5, k)
    dy = 1e-3 / np.sqrt(w)
    y = 1 + dy * rng.normal(0, 1, n) * rng.choice([1, 3])
    y[:k] = 1 + rng.normal(0, 1e-3, k) * 10 ** rng.uniform(-3, 1)
    return t, y, dy


def _narrow_start(seed):
    """The same within the 38-bit encoding: 30 times the others' weight."""
    t, y, dy = _heavy_start(seed)
    heavy = t < 0.05
    dy = np.where(heavy, 1e-3 / np.sqrt(30.0), 1e-3)
    return t, y, dy


@pytest.mark.parametrize("objective", [0, 1], ids=["snr", "likelihood"])
@pytest.mark.parametrize("seeds", [(1030, 2010, 2022, 3051), (3002, 4023, 4052, 4056),
                                   (5009, 8040, 12008, 12046), (6039, 10010, 11027, 15057)])
@pytest.mark.parametrize("make", [_heavy_start, _narrow_start], ids=["heavy", "narrow"])
def test_equals_every_box_in_fp64(make, seeds, objective):
    from cuperiod_b200 import _lib
    periods = 1.0 / np.linspace(1.0 / 20.0, 1.0 / 0.7, 20000)
    grid = _lib.PackedGrid.from_segments([(periods, DURATIONS)], 10, objective)
    curves = _lib.PackedCurves.from_arrays([make(s) for s in seeds])
    out = []
    for exact in (False, True):
        eng = _lib.Engine(exact_sweep=exact)
        eng.prepare(grid, curves)
        eng.launch()
        out.append(np.array(eng.download()))
        eng.close()
    assert np.array_equal(out[0], out[1])
