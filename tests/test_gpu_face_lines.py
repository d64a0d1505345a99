"""The face tables' conveyance along a face's line on the GPU, against the oracle's tables (pinned bit for bit to the
reference): every entry within one float32 ulp, as the device's double cbrt and pow may differ from glibc's in the last
bit. Rough beds, so that a line holds many wet stretches at most levels; the fewest and most pixels a cell and table
rows; lined pixels and crests; lines so long that fewer faces share a CTA's line, and one beyond shared memory."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_tables import FIELDS, ulps
from wadi2d_b200.config import Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.tables import ArrayBed, CrestFaces, build_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "k, rows, reach, edited",
    [(1, 4, 9, False), (3, 33, 20, True), (5, 16, 145, False), (32, 64, 12, True), (32, 4, 5480, False),
     (2, 4, 6400, False)],
    ids=["one_pixel", "odd_rows", "long_reach", "most_pixels", "sixteen_faces", "line_beyond_shared_memory"],
)  # fmt: skip
def test_face_tables_match_the_oracle(k, rows, reach, edited):
    n = 25
    og = O.Grid.from_mask(np.ones((n, n), bool), 0.0, 0.0, 1.0)
    pixel = 144.0 / reach  # the reach past a face's ends is 9 * 16 m in pixels
    dx = k * pixel
    og.dx = dx
    rng = np.random.default_rng(k * 100 + rows)
    side = og.shape[0] * k
    wide = max(side, reach + 1)
    z = 50.0 + 6.0 * rng.standard_normal((side, wide)) + 0.02 * np.arange(wide)[None, :]
    crest, given, npix = None, None, None
    if edited:
        crest, given = O.Crest.empty(og.shape), CrestFaces.empty(og.shape)
        for name in ("xz", "yz"):
            at = rng.random(og.shape) < 0.1
            v = np.where(at, 52.0 + 3.0 * rng.random(og.shape), np.nan)
            setattr(crest, name, v)
            setattr(given, name, v)
        npix = np.where(rng.random(z.shape) < 0.2, 0.02, np.nan)
    ref = O.build_tables(og, z, pixel, 0.035, crest, rows=rows, npix=npix)
    grid = TileGrid(og.x0, og.y0, dx, og.mask)
    got = build_tables(grid, ArrayBed(z, pixel), Tables(rows=rows), 0.035, crest=given, npix=npix)
    for f in FIELDS:
        a, b = getattr(got, f), ref[f]
        assert a.shape == b.shape, f
        assert ulps(a, b).max() <= 1, (f, float(ulps(a, b).max()))
