"""A state written over one that has run: the tiles that had woken sleep again, and the run is the one a fresh model gives,
whatever the first run left in the other halves of the pairs."""

from __future__ import annotations

import numpy as np
import pytest

from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.model import Model
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu
NAMES = ("h", "d", "u", "v", "mx", "my", "qx", "qy", "res", "om")


def _model():
    grid = TileGrid.from_mask(np.ones((60, 700), bool), 0.0, 0.0, 10.0)
    rng = np.random.default_rng(3)
    k = 2
    z = 20.0 - 0.04 * np.arange(grid.shape[1] * k)[None, :] + 0.1 * rng.random((grid.shape[0] * k, grid.shape[1] * k))
    m = Model(build_tables(grid, ArrayBed(z, 5.0), Tables(face_conveyance="strips")), Numerics())
    depth = np.zeros(grid.shape)
    depth[1:59, 1:50] = 2.0
    m.set_depth(depth)
    return m


@pytest.mark.parametrize("host", [False, True], ids=["device", "host"])
@pytest.mark.parametrize("first", [900, 901])
def test_a_rewritten_state_forgets_the_run_before(host, first):
    def go(m, n):
        if host:
            left = [n]

            def count(st):
                left[0] -= 1
                if left[0] == 0:
                    raise StopIteration

            with pytest.raises(StopIteration):
                m.stepper.advance(1e9, on_step=count)
        else:
            m.run(1e9, max_steps=n)

    fresh, used = _model(), _model()
    b, st = used.backend, used.stepper
    start = {name: b.get_field(name).copy() for name in NAMES}
    wet, tiles = b.wet_flags().copy(), b.active_tiles.copy()
    clock = st.t, st.dt, st.nsteps, st.refresh_due
    go(used, first)
    assert b.active_tiles.size > tiles.size + 4  # tiles have woken
    for name in NAMES:
        b.set_field(name, start[name])
    b.wet[:] = wet
    st.t, st.dt, st.nsteps, st.refresh_due = clock
    st.idle[:] = 0
    b.set_active(tiles)
    go(fresh, 300)
    go(used, 300)
    assert fresh.backend.active_tiles.size > tiles.size
    assert st.t == fresh.stepper.t
    for name in NAMES:
        assert np.array_equal(b.get_field(name), fresh.backend.get_field(name)), name
