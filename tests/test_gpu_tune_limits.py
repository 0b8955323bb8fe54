"""BlsTune.smem_per_cta over the whole range that has been taken: up to the device's 227 KB
less 1,552 bytes, whatever the kernels' own static state; more is refused."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _search(weights, **tune):
    from cuperiod_b200 import _lib
    rng = np.random.default_rng(1)
    t = np.sort(rng.uniform(0.0, 30.0, 700))
    y = 1.0 + rng.normal(0.0, 1e-3, t.size)
    y[np.mod(t, 2.3) < 0.1] -= 3e-3
    dy = None if weights == "one" else 1e-3 * rng.uniform(0.7, 1.4, t.size)
    grid = _lib.PackedGrid.from_segments([(np.geomspace(0.7, 5.0, 300), np.array([0.05, 0.1]))],
                                         10, 0)
    eng = _lib.Engine(**tune)
    try:
        return np.array(eng.search(grid, _lib.PackedCurves.from_arrays([(t, y, dy)])))
    finally:
        eng.close()


@pytest.mark.parametrize("weights", ["one", "narrow"])
@pytest.mark.parametrize("smem", [232448 - 1552, 230400, 229000, 228208, 228000])
def test_requests_near_the_limit(weights, smem):
    assert np.array_equal(_search(weights, smem_per_cta=smem), _search(weights))


@pytest.mark.parametrize("smem", [232448 - 1551, 232448, 300000])
def test_requests_past_the_limit(smem):
    from cuperiod_b200.errors import BackendUnavailableError
    with pytest.raises(BackendUnavailableError):
        _search("one", smem_per_cta=smem)
