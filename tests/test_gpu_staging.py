"""The host side of a search: the per-period tables filled in pieces (8,192 periods) by several
threads, and spectra brought back through pinned slots (1 MiB) by several threads.

A segment cut into shorter ones of the same durations has the same phase bins, and box sums are
exact integers, so the spectra must be equal to the last bit; so must a batch's spectra be
however they are downloaded."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DURATIONS = np.array([0.05, 0.08, 0.12])


def _curve(rng, n=250):
    t = np.sort(rng.uniform(0.0, 40.0, n))
    y = 1.0 + rng.normal(0.0, 1e-3, n)
    y[np.mod(t - 0.4, 2.7) < 0.1] -= 4e-3
    return t, y, rng.uniform(0.5e-3, 1.5e-3, n)


def _grid(periods, cuts):
    from cuperiod_b200 import _lib
    return _lib.PackedGrid.from_segments([(p, DURATIONS) for p in np.split(periods, cuts)], 5, 0)


@pytest.mark.parametrize("n", [1, 511, 512, 8192, 8193, 24577])
@pytest.mark.parametrize("descending", [False, True])
def test_pieces_of_a_segment(n, descending):
    from cuperiod_b200 import _lib
    rng = np.random.default_rng(n)
    curves = _lib.PackedCurves.from_arrays([_curve(rng) for _ in range(3)])
    periods = np.geomspace(0.8, 9.0, n)
    if descending:
        periods = periods[::-1].copy()
    eng = _lib.default_engine()
    eng.prepare(_grid(periods, []), curves)
    eng.launch()
    whole = eng.download()
    singly = eng.download_curves(np.arange(3))
    assert whole.shape == (7, 3, n)
    for c in range(3):
        np.testing.assert_array_equal(singly[c], whole[:, c])
    eng.launch()                        # a second launch goes through the graph
    np.testing.assert_array_equal(eng.download(), whole)
    if n > 2:
        # (the widest period sets the fold's fraction bits, not the bins)
        eng.prepare(_grid(periods, sorted({n // 3, n // 2, n - 1})), curves)
        eng.launch()
        np.testing.assert_array_equal(eng.download(), whole)


@pytest.mark.parametrize("where", [0, 8191, 8192, 20000])
@pytest.mark.parametrize("value", [np.nan, np.inf, 0.0, -1.0])
def test_bad_period_in_any_piece(where, value):
    from cuperiod_b200 import _lib
    periods = np.linspace(1.0, 2.0, 20001)
    periods[where] = value
    curves = _lib.PackedCurves.from_arrays([_curve(np.random.default_rng(0))])
    with pytest.raises(ValueError, match="periods must be finite"):
        _lib.default_engine().prepare(_grid(periods, []), curves)
