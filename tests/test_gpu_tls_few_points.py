"""The TLS sweep on either side of the point count from which it estimates a residue before
it divides (80), against the oracle with the bounds of test_gpu_tls."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_tls import _curve
from test_gpu_tls_sizes import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_dur", [3, 5, 9])
@pytest.mark.parametrize("n", [64, 79, 80, 81])
def test_point_counts_around_the_estimate(n, n_dur):
    _check(*_curve(n, n), np.geomspace(0.7, 9.0, 300), n_dur=n_dur)
