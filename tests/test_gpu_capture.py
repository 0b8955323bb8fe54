"""Preparing and launching a search inside a stream capture of the caller's."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _curves(seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(3):
        t = np.sort(rng.uniform(0.0, 30.0, 800))
        y = 1.0 + rng.normal(0.0, 1e-3, t.size)
        y[np.mod(t, 2.3) < 0.1] -= 3e-3
        out.append((t, y, None))
    return out


def test_prepare_and_launch_in_a_capture():
    import torch

    from cuperiod_b200 import _lib
    grid = _lib.PackedGrid.from_segments([(np.geomspace(0.7, 5.0, 500), np.array([0.05, 0.1]))],
                                         10, 0)
    first, second = (_lib.PackedCurves.from_arrays(_curves(s)) for s in (1, 2))
    eng = _lib.Engine(use_graph=False)
    want = {}
    for name, curves in (("second", second), ("first", first)):    # buffers as large as needed
        eng.prepare(grid, curves)
        eng.launch()
        want[name] = np.array(eng.download())
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        eng.prepare(grid, second, stream=stream.cuda_stream)
        eng.launch(stream.cuda_stream)
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(eng.download(), want["second"])
    # and outside of it again
    eng.prepare(grid, first)
    eng.launch()
    assert np.array_equal(eng.download(), want["first"])
    eng.close()


def test_prepare_while_another_stream_captures():
    import torch

    from cuperiod_b200 import _lib
    grid = _lib.PackedGrid.from_segments([(np.geomspace(0.7, 5.0, 500), np.array([0.05, 0.1]))],
                                         10, 0)
    curves = _lib.PackedCurves.from_arrays(_curves(3))
    eng = _lib.Engine()
    eng.prepare(grid, curves)
    eng.launch()
    want = np.array(eng.download())
    x, graph = torch.zeros(4, device="cuda"), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x += 1.0
        eng.prepare(grid, curves)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 1.0
    eng.launch()
    assert np.array_equal(eng.download(), want)
    eng.close()
