"""Places taken ahead (strips 8 at a time, update tiles in a ring of two times 16): a batch that gives a CTA more of them
than it holds, with runs that end on the way, steps as in a launch that gives a CTA a few."""

from __future__ import annotations

import numpy as np
import pytest

from wadi2d_b200 import workloads
from wadi2d_b200.batch import Batch
from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu
RUNS = 310  # 16 tiles each: 4,960, 34 a CTA with one CTA a SM


@pytest.mark.parametrize("steps", [1, 3])
def test_long_lists_and_odd_launches(steps):
    c = workloads.catchment(n=126, dx=10.0, k=2, seed=3, device="cuda")
    grid = TileGrid.from_mask(np.ones((126, 126), bool), 0.0, 0.0, 10.0)
    tables = build_tables(grid, ArrayBed(c.z, 5.0), Tables(), c.manning, device="cuda")
    t_end = np.where(np.arange(RUNS) % 3 == 0, 1.5, 1e9)

    def run(strips, faces, update, per_graph):
        B = Batch([grid] * RUNS, [tables] * RUNS, Numerics())
        B.set_depth([np.full(grid.shape, 0.2 + 0.001 * r) for r in range(RUNS)])
        B.backend.set_loop(False, faces, update, per_graph, strips=strips)
        B.advance(t_end, max_steps=7)
        return [B.field(r, f) for r in range(0, RUNS, 7) for f in ("h", "u", "v", "qx")], B.t.copy(), B.nsteps.copy()

    few, t, n = run(16, 4, 4, 16)
    many, t2, n2 = run(8, 1, 1, steps)
    assert np.array_equal(t, t2) and np.array_equal(n, n2)
    assert n.min() < n.max() == 7
    for a, b in zip(few, many, strict=True):
        assert np.array_equal(a, b)
