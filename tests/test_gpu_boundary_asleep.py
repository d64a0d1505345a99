"""Boundary cells in a tile that is not stepped (no keep flag holds it awake): fixed, free and following ones are
prescribed after every step all the same, whichever form the step takes: the device loop's kernels of their own and its
resident loop at every strip height, a host-driven step as one launch and as kernels of its own."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from wadi2d_b200 import _lib
from wadi2d_b200.backend import BoundaryCells
from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.model import Model
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu
FIELDS = ("h", "d", "u", "v", "qx", "qy", "res", "om")


def _model(kinds):
    """Water in the first tiles of a long basin, boundary cells there and in a tile far away, which sleeps."""
    grid = TileGrid.from_mask(np.ones((40, 500), bool), 0.0, 0.0, 10.0)
    rng = np.random.default_rng(8)
    z = 0.2 * rng.random((grid.shape[0] * 2, grid.shape[1] * 2))
    m = Model(build_tables(grid, ArrayBed(z, 5.0), Tables(face_conveyance="strips")), Numerics())
    depth = np.zeros(grid.shape)
    depth[2:38, 2:20] = 0.5
    m.set_depth(depth)
    index = lambda j, i: m.cell_state_index(j, i)  # noqa: E731
    at = [(j, i) for i in (3, 450) for j in range(4, 36, 2)]
    cell = np.array([index(j, i) for j, i in at], np.int32)
    ref = np.array([index(j, i + 2) for j, i in at], np.int32)
    n = len(at)
    ref[-1] = cell[-1]  # one that follows itself, where kinds has it
    far = cell[n // 2 :]
    m.backend.h[far] = np.linspace(0.1, 0.3, far.size)
    m.backend.d[far] = np.linspace(0.2, 0.5, far.size)
    d0, h0 = np.linspace(0.3, 0.6, n).astype(np.float32), np.linspace(0.1, 0.4, n).astype(np.float32)
    # the backend's own call: Model.set_boundary would keep the boundary tiles awake
    m.backend.set_boundary(BoundaryCells(cell, ref, np.array(kinds, np.int32)[(np.arange(n) + 1) % len(kinds)], d0, h0))
    tile = int(far[0]) // 1296
    assert tile not in m.backend.active_tiles
    return m, tile


def _state(m):
    b = m.backend
    out = [b.get_field(f) for f in FIELDS] + [e.cpu().numpy() for e in b.envelope()]
    return out + [pair[half].cpu().numpy() for pair in (b._t["h"],) for half in (0, 1)]


@pytest.mark.parametrize("kinds", [(0, 1), (0, 1, 2)], ids=["own", "follow"])
@pytest.mark.parametrize("rows", [16, 8, 4])
@pytest.mark.parametrize("arith", ["exact", "fast"])
def test_the_loops_forms_agree(arith, rows, kinds):
    def go(resident: bool):
        m, tile = _model(kinds)
        b = m.backend
        m.backend._params.arith = _lib.ARITH[arith]
        _lib.call("w2b_set_params", b.handle, ctypes.byref(b._params))
        strips = rows if resident else 8
        occ = b.loop_config()[f"{'resident' if resident else 'strips'}{strips}_occupancy"]
        b.set_loop(False, occ, 1, 16, strips=strips, resident=resident)
        states = []
        for steps in (1, 6, 12):
            m.stepper.run(1e9, max_every=2, max_steps=steps)
            assert tile not in b.active_tiles
            states += _state(m)
        return states

    for a, b in zip(go(False), go(True), strict=True):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kinds", [(0, 1), (0, 1, 2)], ids=["own", "follow"])
def test_host_steps_agree(kinds):
    def go(timed: bool):
        m, tile = _model(kinds)
        b, ms = m.backend, (ctypes.c_float * 3)()
        for s in range(7):
            if timed:  # kernels of their own
                _lib.call("w2b_step_timed", b.handle, 0.2, int(s % 4 == 0), 0, b._stream(), ms)
            else:
                b.step(0.2, s % 4 == 0, False)
        return _state(m)

    for a, b in zip(go(True), go(False), strict=True):
        assert np.array_equal(a, b)


def test_cells_set_again():
    """Sets with and without following cells, one after the other, and none."""

    def go(timed: bool):
        m, _ = _model((0, 1, 2))
        b, ms, states = m.backend, (ctypes.c_float * 3)(), []
        every = b.bc
        few = np.nonzero(every.kind < 2)[0]
        own = BoundaryCells(*(getattr(every, f)[few] for f in ("cell", "ref", "kind", "d0", "h0")))
        for bc in (every, own, BoundaryCells.empty(), every):
            b.set_boundary(bc)
            for s in range(3):
                if timed:
                    _lib.call("w2b_step_timed", b.handle, 0.2, int(s == 0), 0, b._stream(), ms)
                else:
                    b.step(0.2, s == 0, False)
            states += _state(m)
        return states

    for a, b in zip(go(True), go(False), strict=True):
        assert np.array_equal(a, b)
