"""A prepare leaves alone the staging memory of uploads that still wait on the stream: with
work queued ahead, a star (or a set of curves) is prepared and launched, the next one is
prepared, and what the launch wrote is the first one's."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PERIODS = np.geomspace(0.7, 5.0, 600)


def _curve(rng, n=900):
    t = np.sort(rng.uniform(0.0, 30.0, n))
    t[0], t[-1] = 0.0, 30.0
    y = 1.0 + rng.normal(0.0, 1e-3, n)
    y[np.mod(t, rng.uniform(1.0, 3.0)) < 0.1] -= 3e-3
    return t, y, 1e-3 * rng.uniform(0.7, 1.4, n)


def _joint(eng, seed):
    from cuperiod_b200 import _lib
    rng = np.random.default_rng(seed)
    grid = _lib.PackedGrid.from_segments([(PERIODS, np.array([0.05, 0.1]))], 10, 0)
    bands = _lib.PackedCurves.from_arrays([_curve(rng) for _ in range(3)])
    return (lambda s=None: eng.joint_prepare(grid, bands, s), eng.joint_launch,
            eng.joint_download)


def _tls(eng, seed):
    from cuperiod_b200 import tls
    rng = np.random.default_rng(seed)
    curves = [tls._prepare(*_curve(rng))[0] for _ in range(3)]
    widths = [3, 6, 11, 20]
    templates = {d: tls.limb_darkened_template(d, 0.4, 0.3) for d in widths}
    return (lambda s=None: eng.tls_prepare(curves, PERIODS, n_bins=200, dur_bins=widths,
                                           templates=templates, den_rel=1e-9, stream=s),
            eng.tls_launch, eng.tls_download)


@pytest.mark.parametrize("search", [_joint, _tls], ids=["joint", "tls"])
def test_a_queued_upload_keeps_its_inputs(search):
    import torch

    from cuperiod_b200 import _lib
    eng = _lib.Engine()
    want = []
    for seed in (1, 2):
        prepare, launch, download = search(eng, seed)
        prepare()
        launch()
        want.append(np.array(download()))
    assert not np.array_equal(want[0], want[1])
    stream = torch.cuda.Stream()
    s = stream.cuda_stream
    first, second = search(eng, 1), search(eng, 2)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(200_000_000)          # about a tenth of a second
    first[0](s)
    first[1](s)
    second[0](s)
    assert np.array_equal(first[2](s), want[0])
    second[1](s)
    assert np.array_equal(second[2](s), want[1])
    eng.close()
