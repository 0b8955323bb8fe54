"""The TLS matched filter in any unit of the flux: with the flux in units 2^k times larger,
every sum scales by a power of two, which FP64 carries exactly, so the signal residue, the
duration and the epoch are the same bits and the depth is 2^k times larger."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_BINS = 200
WIDTHS = [3, 6, 11, 20, 37, 60]


@pytest.fixture(scope="module")
def engine():
    from cuperiod_b200 import _lib
    eng = _lib.Engine()
    yield eng
    eng.close()


@pytest.fixture(scope="module")
def search(engine):
    from cuperiod_b200 import tls
    rng = np.random.default_rng(3)
    n = 500
    tau = np.sort(rng.uniform(0.0, 60.0, n))
    tau -= tau[0]
    y = rng.normal(0.0, 1.0, n)
    y[np.mod(tau, 3.1) < 0.4] -= 2.0
    w = 1.0 / rng.uniform(0.7, 1.4, n) ** 2
    w_total = float(w.sum())
    yw = w * (y - float(np.dot(w, y) / w_total))
    periods = np.geomspace(0.8, 12.0, 400)
    templates = {d: tls.limb_darkened_template(d, 0.4, 0.3) for d in WIDTHS}

    def run(k):
        curve = (tau, yw * 2.0 ** -k, w * 2.0 ** (-2 * k), w_total * 2.0 ** (-2 * k))
        return engine.tls_search([curve], periods, n_bins=N_BINS, dur_bins=WIDTHS,
                                 templates=templates, den_rel=1e-9)
    return run


@pytest.mark.parametrize("k", [-200, -70, -60, -50, -20, 20, 35, 38, 40, 42, 44, 46, 48, 50, 52, 55, 60,
                               200])
def test_units_of_the_flux(search, k):
    sr, depth, duration, t0 = search(0)
    got = search(k)
    assert np.array_equal(got[0], sr)
    assert np.array_equal(got[1], depth * 2.0 ** k)
    assert np.array_equal(got[2], duration)
    assert np.array_equal(got[3], t0)
