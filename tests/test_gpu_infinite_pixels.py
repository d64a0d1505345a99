"""Infinite pixels (walls, holes) in a face's line: the face tables are the oracle's, whose running sums carry what is not
finite in them along the line."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_tables import FIELDS, ulps
from wadi2d_b200.config import Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("k, rows", [(1, 16), (3, 33), (5, 4), (16, 16)])
@pytest.mark.parametrize("share", [0.02, 0.0005])
def test_face_tables_match_the_oracle(value, k, rows, share):
    n = 25
    og = O.Grid.from_mask(np.ones((n, n), bool), 0.0, 0.0, 10.0)
    rng = np.random.default_rng(k)
    z = 50.0 + 6.0 * rng.standard_normal((og.shape[0] * k, og.shape[1] * k))
    z[rng.random(z.shape) < share] = value
    z[z.shape[0] // 2, z.shape[1] // 2] = value
    with np.errstate(all="ignore"):
        ref = O.build_tables(og, z, 10.0 / k, 0.035, None, rows=rows)
    grid = TileGrid(og.x0, og.y0, 10.0, og.mask)
    got = build_tables(grid, ArrayBed(z, 10.0 / k), Tables(rows=rows), 0.035)
    for f in ("efx", "efy", "ftabx", "ftaby"):
        a, b = getattr(got, f), ref[f]
        assert f in FIELDS and np.array_equal(np.isfinite(a), np.isfinite(b)), f
        good = np.isfinite(b)
        assert good.any() and ulps(a[good], b[good]).max() <= 1, (f, float(ulps(a[good], b[good]).max()))
