"""The device's peak ranking on either side of the grid size from which the candidates' bitmap
leaves no room for the list of the best (917,504 periods): the same total order, as
test_gpu_row_lists restates it."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_row_lists import _check
from test_gpu_rows import engine  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_periods", [917_504, 917_505])
def test_peaks_around_the_lists_limit(engine, n_periods):  # noqa: F811
    rng = np.random.default_rng(n_periods)
    t = np.sort(rng.uniform(0.0, 40.0, 60))
    y = 1.0 + rng.normal(0.0, 1e-3, t.size)
    y[np.mod(t, 2.7) < 0.3] -= 4e-3
    _check(engine, [(t, y, np.full(t.size, 1e-3))], n_periods, 10, 0.0035, 8, 0.1)
