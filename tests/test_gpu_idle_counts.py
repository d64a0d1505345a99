"""The idle counts that a program took from the stepper before a run: the array keeps the counts, and what is written into it
goes to the next run."""

from __future__ import annotations

import numpy as np
import pytest

from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.model import Model
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu


def test_an_array_taken_before_the_run():
    grid = TileGrid.from_mask(np.ones((60, 500), bool), 0.0, 0.0, 10.0)
    z = 0.3 * np.random.default_rng(4).random((grid.shape[0] * 2, grid.shape[1] * 2))
    m = Model(build_tables(grid, ArrayBed(z, 5.0), Tables(face_conveyance="strips")), Numerics())
    depth = np.zeros(grid.shape)
    depth[1:61, 1:60] = 0.4
    m.set_depth(depth)
    device = m.backend._t["idle"]
    held = m.stepper.idle
    m.run(1e9, max_steps=40)
    assert held.any() and np.array_equal(held, device.cpu().numpy())
    held[1:] = 7
    m.run(1e9, max_steps=1)  # no check falls on this step
    assert np.array_equal(held[1:], np.full(held.size - 1, 7, np.int32))
    assert np.array_equal(m.stepper.idle, device.cpu().numpy())
