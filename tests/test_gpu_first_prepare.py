"""The work plan of a batch does not depend on what the process has searched before: the first
prepare of a fresh process cuts the same tiles as a later one of the same batch."""

from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import numpy as np
from cuperiod_b200 import _lib
rng = np.random.default_rng(1)
t = np.sort(rng.uniform(0.0, 60.0, 300))
curves = _lib.PackedCurves.from_arrays([(t, 1.0 + rng.normal(0.0, 1e-3, t.size), {errors})])
grid = _lib.PackedGrid.from_segments([(np.geomspace(0.6, 8.0, 1000), np.array([0.05, 0.1]))], 10, 0)
items = []
for _ in range(2):
    eng = _lib.Engine()
    eng.prepare(grid, curves)
    items.append(eng.info()["n_items"])
    eng.close()
print(*items)
"""


@pytest.mark.parametrize("errors", ["None", "1e-3 * rng.uniform(0.7, 1.4, t.size)"],
                         ids=["one", "narrow"])
def test_first_and_later_plans_are_the_same(errors):
    out = subprocess.run([sys.executable, "-c", PROGRAM.format(errors=errors)], cwd=ROOT,
                         capture_output=True, text=True, timeout=300, check=True)
    first, later = map(int, out.stdout.split())
    assert first == later
