"""The resident loop (several steps in one cooperative launch) against the loop's kernels of their own, bit for bit: the
golden cases (rain, free outfall, sleeping tiles, envelope and tally; fixed stages, following boundary cells, crests and
tiles that wake) in both builds and with every strip height, launches that end inside a run, and a batch whose runs stop
at different steps."""

from __future__ import annotations

import numpy as np
import pytest

import cases
from product_api import B200Api
from wadi2d_b200.batch import Batch
from wadi2d_b200.config import Numerics
from wadi2d_b200.tables import ArrayBed, build_tables
from wadi2d_b200.config import Tables
from wadi2d_b200.grid import TileGrid

pytestmark = pytest.mark.gpu


def _fix(backend, resident: bool, rows: int, steps: int) -> None:
    cfg = backend.loop_config()
    kind = "resident" if resident else "strips"
    backend.set_loop(False, cfg[f"{kind}{rows}_occupancy"], 1, steps, strips=rows, resident=resident)
    assert backend.loop_config()["resident"] == int(resident)


class FixedApi(B200Api):
    def __init__(self, resident: bool, rows: int, steps: int, arith: str) -> None:
        super().__init__(device_loop=True, arith=arith)
        self.form = (resident, rows, steps)

    def model(self, grid, tables, numerics):
        m = super().model(grid, tables, numerics)
        _fix(m.backend, *self.form)
        return m


@pytest.mark.parametrize("steps", [1, 7, 32])
@pytest.mark.parametrize("rows", [16, 8, 4])
@pytest.mark.parametrize("arith", ["exact", "fast"])
@pytest.mark.parametrize("case", list(cases.CASES))
def test_resident_loop_equals_the_kernels_of_their_own(case, arith, rows, steps):
    a, _ = cases.CASES[case](FixedApi(False, 8, 16, arith))
    b, _ = cases.CASES[case](FixedApi(True, rows, steps, arith))
    for key in a:
        assert np.array_equal(np.asarray(a[key]), np.asarray(b[key]), equal_nan=True), key


def _batch(resident: bool, rows: int):
    rng = np.random.default_rng(3)
    sides, ends = (40, 75, 33, 98), (60.0, 200.0, 25.0, 120.0)
    tabs = []
    for r, n in enumerate(sides):
        grid = TileGrid.from_mask(np.ones((n, n), bool), 0.0, 0.0, 8.0 + r)
        z = 0.02 * np.arange(grid.shape[1] * 4)[None, :] + 0.4 * rng.random((grid.shape[0] * 4, grid.shape[1] * 4))
        tabs.append(build_tables(grid, ArrayBed(z, (8.0 + r) / 4), Tables()))
    B = Batch([t.grid for t in tabs], tabs, Numerics())
    _fix(B.backend, resident, rows, 16)
    B.set_depth([np.where(t.grid.mask, 0.3 * (r % 2) + 0.05, 0.0) for r, t in enumerate(tabs)])
    B.set_source([np.where(t.grid.mask, 1e-5 * (r + 1), 0.0) for r, t in enumerate(tabs)])
    B.advance(np.array(ends), max_every=4)
    out = [B.t.copy(), B.dt.copy(), B.nsteps.copy()]
    for r in range(len(sides)):
        out += [B.field(r, f) for f in ("h", "d", "u", "v", "qx", "qy", "res")] + list(B.envelope(r).values())
    return out


@pytest.mark.parametrize("rows", [16, 8, 4])
def test_resident_loop_steps_a_batch_whose_runs_stop_apart(rows):
    a, b = _batch(False, 8), _batch(True, rows)
    assert len(set(a[2].tolist())) > 1
    for x, y in zip(a, b, strict=True):
        assert np.array_equal(x, y)
