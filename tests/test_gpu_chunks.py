"""The device loop's launches of fewer steps at the end of a call (graphs of 4 steps and of 1 beside the configuration's),
and the lists read back when asked for: a run in calls of every length around them equals the same run in one call, bit for
bit, and the host's active list and idle counts are the device's."""

from __future__ import annotations

import numpy as np
import pytest

from wadi2d_b200 import workloads
from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.model import Model
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu

CALLS = (1, 3, 4, 5, 16, 17, 21, 47, 130)


def _model(form):
    w = workloads.v_channel_plane(n=90, dx=10.0, k=4, seed=2)
    grid = TileGrid.from_mask(np.ones((90, 90), bool), 0.0, 0.0, w.dx)
    m = Model(build_tables(grid, ArrayBed(w.z, w.dx / w.k), Tables(), w.manning), Numerics())
    depth = np.zeros(grid.shape)
    depth[20:40, 20:60] = 0.4  # the rest dry, most tiles asleep at first
    m.set_depth(depth)
    if form is not None:
        cfg = m.backend.loop_config()
        rows, resident = form
        kind = "resident" if resident else "strips"
        m.backend.set_loop(False, cfg[f"{kind}{rows}_occupancy"], 1, 16, strips=rows, resident=resident)
    return m


@pytest.mark.parametrize("form", [(8, False), (8, True)], ids=["graphs", "resident"])
def test_calls_of_any_length_are_one_run(form):
    whole, parts = _model(form), _model(form)
    whole.run(1e9, max_steps=sum(CALLS))
    done = 0
    for n in CALLS:
        parts.run(1e9, max_steps=n)
        done += n
        assert parts.stepper.nsteps == done
    assert parts.stepper.t == whole.stepper.t and parts.stepper.dt == whole.stepper.dt
    for name in ("h", "d", "u", "v", "qx", "qy", "res", "om"):
        assert np.array_equal(parts.backend.get_field(name), whole.backend.get_field(name)), name
    # windows end on time, whatever the step rule does on the way
    for k in range(1, 5):
        assert parts.run(parts.stepper.t + 7.3 * k) == pytest.approx(parts.stepper.t, abs=1e-9)


def test_lists_are_the_devices():
    m = _model((8, True))
    b = m.backend
    for n in (20, 60, 200):
        m.run(1e9, max_steps=n)
        nact = int(b.nact)
        assert np.array_equal(b.active_tiles, b._t["active"][:nact].cpu().numpy())
        assert np.array_equal(m.stepper.idle, b._t["idle"].cpu().numpy())
    tiles = b.active_tiles
    # a list the caller changed in place is sent all the same
    fewer = tiles.copy()
    b.set_active(fewer)
    fewer[-1] = fewer[0]
    b.set_active(fewer)
    assert np.array_equal(b._t["active"][: fewer.size].cpu().numpy(), fewer)
    flags = np.zeros(m.grid.ntiles, np.int32)
    flags[fewer] = 1
    assert np.array_equal(b._t["is_act"].cpu().numpy(), flags)


def test_host_steps_in_one_launch_equal_the_kernels_of_their_own():
    """A grid small enough for one launch a step against a batch-sized one (the same run with a dry block of tiles beside
    it that lifts it over the line), with fixed, free and following boundary cells."""
    from wadi2d_b200.backend import BoundaryCells

    def run(wide: bool):
        n, m = 60, 60
        grid = TileGrid.from_mask(np.ones((n, m if not wide else 4000), bool), 0.0, 0.0, 10.0)
        k = 2
        rng = np.random.default_rng(5)
        z = np.full((grid.shape[0] * k, grid.shape[1] * k), 50.0)
        z[: 64 * k, : 61 * k] = 0.05 * np.arange(61 * k)[None, ::-1] + 0.3 * rng.random((64 * k, 61 * k))
        model = Model(build_tables(grid, ArrayBed(z, 5.0), Tables(face_conveyance="strips")), Numerics())
        model.stepper.adaptive_active = False
        depth = np.zeros(grid.shape)
        depth[1:61, 1:61] = 0.4
        model.set_depth(depth)
        rows = np.arange(5, 25)
        cell = np.array([model.cell_state_index(int(j), 1) for j in rows], np.int32)
        ref = np.array([model.cell_state_index(int(j), 3) for j in rows], np.int32)
        kind = np.arange(20, dtype=np.int32) % 3
        model.set_boundary(BoundaryCells(cell, ref, kind, np.full(20, 0.3, np.float32), np.full(20, 0.2, np.float32)))
        for s in range(30):
            model.backend.step(0.4, s % 8 == 0, s % 5 == 0)
        wave = model.backend.max_wave()
        return [model.field(f)[:64, :61] for f in ("h", "d", "u", "v", "qx", "qy", "res")], wave

    small, wide = run(False), run(True)
    assert small[1] == wide[1]
    for a, b in zip(small[0], wide[0], strict=True):
        assert np.array_equal(a, b)
