"""The TLS kernel at the point counts, bin counts and template counts where its fold and
sweep change shape, against the oracle: the same bounds as test_gpu_tls.

Points per block (1,024 or 2,048, and the tail's), samplings on either side of the line
between merged and single adds, templates in groups of four, times whose fast fold is not
provable, and times on bin edges (more than the list of open points holds).
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle
from test_gpu_tls import _agree, _curve

pytestmark = pytest.mark.gpu


def _check(t, y, dy, periods, **kw):
    from cuperiod_b200.settings import TLSSettings
    from cuperiod_b200.tls import tls_power
    got = tls_power(t, y, dy, periods, settings=TLSSettings(**{
        "n_phase_bins": kw.get("n_bins", 256), "n_durations": kw.get("n_dur", 5)}))
    ref = oracle.tls_power(t, y, dy, periods, n_bins=kw.get("n_bins", 256),
                           n_durations=kw.get("n_dur", 5), n_threads=8)
    _agree(got, ref, min_same=0.98)


@pytest.mark.parametrize("n", [50, 255, 257, 1023, 1025, 2047, 2049, 3071, 3073, 4096])
def test_point_counts(n):
    _check(*_curve(n, n), np.geomspace(0.7, 9.0, 300))


@pytest.mark.parametrize("n_dur", [1, 3, 4, 6, 8, 9])
@pytest.mark.parametrize("n_bins", [16, 31, 256, 300])
def test_template_counts(n_bins, n_dur):
    _check(*_curve(n_dur, 3000), np.geomspace(0.7, 9.0, 200), n_bins=n_bins, n_dur=n_dur)


@pytest.mark.parametrize("span", [2.0, 20.0, 200.0])
def test_sampling_beside_the_bins(span):
    # 6,000 points over 2 days: several per bin; over 200 days: bins finer than the gaps
    _check(*_curve(7, 6000, span=span, period=0.61), np.geomspace(0.3, span / 2.5, 200))


def test_times_on_bin_edges():
    # a cadence that divides the period: every point on an edge, so every bin is the exact
    # path's
    n = 5000
    rng = np.random.default_rng(2)
    t = np.arange(n) / 512.0
    y = 1.0 + rng.normal(0.0, 1e-3, n)
    y[np.mod(t, 2.0) < 0.06] -= 3e-3
    _check(t, y, np.full(n, 1e-3), np.concatenate([[0.5, 1.0, 2.0, 4.0], np.geomspace(0.6, 4.5, 60)]))


def test_fold_without_a_provable_fast_path():
    # 3e5 cycles: past the fast fold's range
    t, y, dy = _curve(3, 2500, span=3000.0, period=0.0098)
    _check(t, y, dy, np.linspace(0.0097, 0.0099, 40))
