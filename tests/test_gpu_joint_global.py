"""The shared-ephemeris kernel with histograms in global memory (more bins times bands than
shared memory holds), whose prefix sums take 32 bins of a run at a time: bands that share the
CTA's warps evenly or not, one run a band, two turns of the warps, runs that end inside 32 bins.
Bounds as in test_gpu_joint_sizes."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_joint import _engine_vs_oracle, _star

pytestmark = pytest.mark.gpu

# bands, bins of the shortest and longest period
CASES = [(1, 13500, 14100), (2, 7200, 7400), (3, 4900, 5000), (5, 3010, 3050), (11, 1400, 1430),
         (17, 900, 960), (32, 510, 600), (33, 511, 513), (64, 255, 290)]


def _case(bands, lo, hi):
    rng = np.random.default_rng(bands)
    span = 60.0
    star = _star(rng, bands, n=(30, 60), span=span)
    bin_ = 0.003
    periods = np.linspace(lo * bin_, hi * bin_, 12)
    durations = bin_ * 10 * np.array([1.0, 2.0, 3.5, 7.0])
    return star, [periods], [durations], 10


@pytest.mark.parametrize("bands,lo,hi", CASES)
def test_snr_power(bands, lo, hi):
    got, ref = _engine_vs_oracle(*_case(bands, lo, hi), 0)
    scale = float(ref["power"].max())
    assert scale > 0.0
    np.testing.assert_allclose(got["power"], ref["power"], rtol=1e-6, atol=1e-9 * scale)
