"""Reading cells (a gauge) between host-driven steps is only a read: the steps do not go over the sleeping tiles for it, as
they do after a write, and their results are the same."""

from __future__ import annotations

import numpy as np
import pytest

from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.layout import native_of_ref
from wadi2d_b200.model import Model
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu


def _model():
    grid = TileGrid.from_mask(np.ones((60, 500), bool), 0.0, 0.0, 10.0)
    z = 0.3 * np.random.default_rng(4).random((grid.shape[0] * 2, grid.shape[1] * 2))
    m = Model(build_tables(grid, ArrayBed(z, 5.0), Tables(face_conveyance="strips")), Numerics())
    depth = np.zeros(grid.shape)
    depth[1:61, 1:60] = np.linspace(0.2, 0.9, 59)[None, :]
    m.set_depth(depth)
    return m


@pytest.mark.parametrize("name", ["h", "u", "v"])
def test_a_read_leaves_the_sleeping_tiles_alone(name):
    m = _model()
    b = m.backend
    gauge = np.array([m.cell_state_index(30, 40)])
    asleep = m.cell_state_index(30, 450)
    assert asleep // 1296 not in b.active_tiles
    b.step(0.2, True, False)  # what set_depth touched is settled
    native = int(native_of_ref(m.grid.tiles, np.array([asleep]), m.grid.shape[1])[0])
    b._t["h"][:, native] = b.torch.tensor([3.0, 5.0], device=b.device)  # halves that differ, behind the library's back
    m.read_cells(name, gauge)
    b.step(0.2, True, False)
    assert sorted(b._t["h"][:, native].tolist()) == [3.0, 5.0]
    getattr(b, name)[gauge] = m.read_cells(name, gauge)  # a write settles them
    b.step(0.2, True, False)
    assert b._t["h"][0, native] == b._t["h"][1, native]


def test_a_gauge_changes_no_step():
    def go(read: bool):
        m = _model()
        gauge = np.array([m.cell_state_index(30, i) for i in (20, 58, 62, 90)])
        seen = []

        def note(st):
            if read:
                seen.append(m.read_cells("h", gauge).copy())
            if st.nsteps == 60:
                raise StopIteration

        with pytest.raises(StopIteration):
            m.advance(1e9, on_step=note)
        return [m.backend.get_field(f) for f in ("h", "d", "u", "v", "qx", "qy", "res")] + [m.read_cells("h", gauge)], seen

    (a, _), (b, seen) = go(False), go(True)
    for x, y in zip(a, b, strict=True):
        assert np.array_equal(x, y)
    assert len(seen) == 60 and np.array_equal(seen[-1], b[-1])
