"""The wave maximum that w2b_max_wave reads after the device loop is the last refresh step's, whichever of the loop's two
sets of settings that step read: after calls of odd and even lengths, against the host loop's own readings, and after
host-driven steps that do not refresh it."""

from __future__ import annotations

import numpy as np
import pytest

from wadi2d_b200 import workloads
from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.model import Model
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu
CALLS = (1, 3, 4, 5, 17, 2, 33, 8, 6)


def _model():
    w = workloads.v_channel_plane(n=90, dx=10.0, k=4, seed=2)
    grid = TileGrid.from_mask(np.ones((90, 90), bool), 0.0, 0.0, w.dx)
    m = Model(build_tables(grid, ArrayBed(w.z, w.dx / w.k), Tables(), w.manning), Numerics())
    depth = np.zeros(grid.shape)
    depth[20:40, 20:60] = 0.4
    m.set_depth(depth)
    return m


def _host_waves(steps: int) -> list:
    """The wave maximum after each host-driven step."""
    m, waves = _model(), []

    def note(st):
        waves.append(st.backend.max_wave())
        if len(waves) == steps:
            raise StopIteration

    with pytest.raises(StopIteration):
        m.advance(1e9, on_step=note)
    return waves


@pytest.mark.parametrize("form", [None, (8, False), (8, True)], ids=["tuning", "graphs", "resident"])
def test_max_wave_after_calls_of_any_length(form):
    waves = _host_waves(sum(CALLS))
    assert len(set(waves)) > 5
    m = _model()
    if form is not None:
        rows, resident = form
        occ = m.backend.loop_config()[f"{'resident' if resident else 'strips'}{rows}_occupancy"]
        m.backend.set_loop(False, occ, 1, 16, strips=rows, resident=resident)
    done = 0
    for n in CALLS:
        m.run(1e9, max_steps=n)
        done += n
        assert m.stepper.nsteps == done
        assert m.backend.max_wave() == waves[done - 1], n
    for _ in range(3):
        m.backend.step(0.01, False, False)
        assert m.backend.max_wave() == waves[-1]
