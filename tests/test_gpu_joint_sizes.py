"""The shared-ephemeris kernel at the sizes where its screen and its layout change: bands of one
to three points (every box empty of a band or full of it), weights too unequal for the screen's
high words, one to thirty-two durations (groups of four with a remainder), periods barely longer
than the wrap pad (pad copied in order) and of several thousand bins, 64 bands.

With the SNR objective a box chosen differently on a tie to rounding has the same power, so every
period's power is compared: the engine's sums carry 2^-61 per point, the oracle's sequential
sums about 2^-52 times the points, and a squared depth SNR amplifies either by no more than
(level / depth) ~ 1e4 here, far inside 1e-6.  The likelihood objective's power is not what is
maximised: there the boxes agree at all but 1% of the periods."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_joint import _agree, _engine_vs_oracle, _star

pytestmark = pytest.mark.gpu


def _grid(n_dur, oversample, periods, shortest=0.03):
    return [np.asarray(periods)], [np.geomspace(shortest, 0.35, n_dur) if n_dur > 1
                                   else np.array([shortest])], oversample


CASES = {
    "points1": (lambda r: _star(r, 1, n=(1, 2)) + _star(r, 2, n=(60, 90)),
                _grid(6, 5, np.geomspace(0.9, 3.0, 150))),
    "points2": (lambda r: _star(r, 3, n=(2, 3)) + _star(r, 1, n=(100, 101)),
                _grid(7, 5, np.geomspace(0.9, 3.0, 150))),
    "points3": (lambda r: _star(r, 5, n=(3, 4)), _grid(5, 10, np.geomspace(0.9, 3.0, 150))),
    "one_duration": (lambda r: _star(r, 2), _grid(1, 3, np.geomspace(0.9, 3.0, 150))),
    "durations32": (lambda r: _star(r, 2), _grid(32, 10, np.geomspace(0.9, 3.0, 150))),
    "short": (lambda r: _star(r, 3), _grid(4, 10, np.geomspace(0.034, 0.07, 200))),
    "long": (lambda r: _star(r, 1), _grid(9, 10, np.geomspace(9.0, 14.0, 60))),
    "bands64": (lambda r: _star(r, 64, n=(5, 40)), _grid(3, 3, np.geomspace(0.9, 1.5, 60))),
    "unequal": (lambda r: [(t, y, dy * np.where(np.arange(t.size) % 7 == 3, 3e5, 1.0))
                           for t, y, dy in _star(r, 3)],
                _grid(5, 5, np.geomspace(0.9, 3.0, 100))),
}


@pytest.mark.parametrize("name", CASES)
def test_snr_power(name):
    make, (periods, durations, oversample) = CASES[name]
    bands = make(np.random.default_rng(len(name)))
    got, ref = _engine_vs_oracle(bands, periods, durations, oversample, 0)
    scale = float(ref["power"].max())
    assert scale > 0.0
    np.testing.assert_allclose(got["power"], ref["power"], rtol=1e-6, atol=1e-9 * scale)
    np.testing.assert_allclose(got["depth_snr"] ** 2, got["power"], rtol=1e-12, atol=0.0)


@pytest.mark.parametrize("name", ["one_duration", "durations32", "long"])
def test_likelihood_boxes(name):
    make, (periods, durations, oversample) = CASES[name]
    bands = make(np.random.default_rng(len(name)))
    got, ref = _engine_vs_oracle(bands, periods, durations, oversample, 1)
    _agree(got, ref)
