"""The device's peak ranking where its list of the best candidates begins and ends: fewer
candidates than the list holds, rows that outlast one list and the next, a score shared by more
candidates than a list holds (the ranking goes on over the bitmap), more harmonics than the
precomputed test has, plateaus of equal powers.  The ranking is a total order (power, then the
candidate's place), so the peaks equal the greedy choice restated here; the host's rows, whose
sort leaves the order of equal scores open, are compared elsewhere."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_rows import _keyed, engine  # noqa: F401

pytestmark = pytest.mark.gpu


def _greedy(power, freq, n_best, tol, hmax, sep):
    from cuperiod_b200.result import is_alias_related
    p = np.where(np.isfinite(power), power, 0.0)
    n = p.size
    cand = [(p[j], n - 1 - j, j) for j in range(1, n - 1) if p[j] > p[j + 1] and p[j] >= p[j - 1]]
    if p[n - 1] >= p[n - 2]:
        cand.append((p[n - 1], n, n - 1))
    if p[0] > p[1]:
        cand.append((p[0], n + 1, 0))
    chosen = []
    for _, _, j in sorted(cand, reverse=True):
        if len(chosen) == n_best:
            break
        if not any(is_alias_related(a, b, tol, hmax, min_separation=sep)
                   for c in chosen for a, b in ((freq[j], freq[c]), (freq[c], freq[j]))):
            chosen.append(j)
    return chosen


def _check(engine, curves, n_periods, n_best, tol, hmax, sep):
    from cuperiod_b200 import _lib
    periods = np.geomspace(0.5, 12.0, n_periods)
    grid = _lib.PackedGrid.from_segments([(periods, np.array([0.03, 0.06]))], 10, 0)
    engine.prepare(grid, _lib.PackedCurves.from_arrays(curves))
    engine.launch()
    power = engine.download()[0]
    n = len(curves)
    count, index, _ = engine.rows(n_best, hmax, np.full(n, sep), np.full(n, tol))
    for c in range(n):
        want = _greedy(power[c], 1.0 / periods, n_best, tol, hmax, sep)
        assert int(count[c]) == len(want)
        np.testing.assert_array_equal(index[c, :len(want)], want)
    return power


@pytest.mark.parametrize("n_periods,n_best,tolerance,harmonics,separation", [
    (600, 40, 0.0035, 8, 0.1),      # every candidate listed
    (20000, 150, 1e-6, 2, 1e-3),    # several lists
    (60000, 10, 0.0035, 8, 0.1),
    (60000, 60, 1e-5, 3, 1e-2),
    (20000, 12, 0.0035, 40, 0.1),
])
def test_peaks(engine, n_periods, n_best, tolerance, harmonics, separation):  # noqa: F811
    curves = [(lc.time, lc.value, lc.error) for _, lc in _keyed()[:4]]
    _check(engine, curves, n_periods, n_best, tolerance, harmonics, separation)


@pytest.mark.parametrize("n_periods,n_best", [(700, 30), (60000, 30)])
def test_plateaus(engine, n_periods, n_best):  # noqa: F811
    rng = np.random.default_rng(n_periods)
    t = np.sort(rng.uniform(0.0, 27.0, 40))
    y = 1.0 - 0.01 * (rng.integers(0, 4, 40) == 0)      # two flux values
    power = _check(engine, [(t, y, np.full(40, 1e-3))], n_periods, n_best, 2e-5, 3, 1e-4)
    assert np.unique(power).size < 0.5 * n_periods
