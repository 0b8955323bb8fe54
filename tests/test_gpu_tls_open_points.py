"""More points on bin edges than the TLS fold's list of open points holds, at every period of
its tiles, against the oracle with the bounds of test_gpu_tls."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_tls_sizes import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [700, 2300, 6200])
def test_every_point_of_every_period_on_an_edge(n):
    # a cadence of 1/512 and periods of whole quarters: full blocks and tails
    t = np.arange(n) / 512.0
    y = 1.0 + np.random.default_rng(n).normal(0.0, 1e-3, n)
    y[np.mod(t, 0.75) < 0.06] -= 3e-3
    _check(t, y, np.full(n, 1e-3), np.arange(1, 25) / 4.0)
