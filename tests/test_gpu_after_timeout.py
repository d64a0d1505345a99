"""After a bounded wait has given up (the status and the grid barrier's counters as such a launch leaves them, written by the
test): no launch that waits at a grid barrier begins, the failure is reported, the device loop begins anew, and the kernels
that count their CTAs without waiting count right."""

from __future__ import annotations

import numpy as np
import pytest

from wadi2d_b200 import _lib
from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.model import Model
from wadi2d_b200.surrogate import Network
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu
STATUS, GRID = 5, 128  # int32 places in the control block: Ctl::status, GridState (arrivals, CTAs that have left)
FIELDS = ("h", "d", "u", "v", "mx", "my", "qx", "qy", "res")


def _model():
    grid = TileGrid.from_mask(np.ones((60, 90), bool), 0.0, 0.0, 10.0)
    z = 0.3 * np.random.default_rng(4).random((grid.shape[0] * 2, grid.shape[1] * 2))
    m = Model(build_tables(grid, ArrayBed(z, 5.0), Tables(face_conveyance="strips")), Numerics())
    depth = np.zeros(grid.shape)
    depth[1:61, 1:91] = np.linspace(0.2, 0.9, 90)[None, :]
    m.set_depth(depth)
    for s in range(5):
        m.backend.step(0.3, s % 4 == 0, False)
    return m


def _plant(m, status: int) -> None:
    words = m.backend._t["ctl"].view(m.backend.torch.int32)
    words[STATUS] = status
    words[GRID], words[GRID + 1] = 3, 2


def _state(m):
    return [m.backend.get_field(f) for f in FIELDS]


@pytest.mark.parametrize("steps", [1, 2])
def test_steps_wait_for_the_failure_to_be_dealt_with(steps):
    m, fresh = _model(), _model()
    b = m.backend
    _plant(m, _lib.ETIMEOUT)
    for _ in range(steps):
        b.step(0.3, True, False)
    for _ in range(2):
        with pytest.raises(_lib.W2BError):
            b.max_wave()
    for x, y in zip(_state(m), _state(fresh), strict=True):
        assert np.array_equal(x, y)
    resident = b.loop_config()["resident8_occupancy"]
    for one in (m, fresh):
        one.backend.set_loop(False, resident, 1, 8, strips=8, resident=True)
        one.run(1e9, max_steps=20)
    for x, y in zip(_state(m), _state(fresh), strict=True):
        assert np.array_equal(x, y)
    assert b.max_wave() == fresh.backend.max_wave()


def test_the_momenta_are_stored_all_the_same():
    m, fresh = _model(), _model()
    _plant(m, 0)
    for one in (m, fresh):
        one.backend.set_field("u", 0.5 * one.backend.get_field("u"))
        _lib.call("w2b_step_timed", one.backend.handle, 0.3, 1, 0, one.backend._stream(), (_lib.c_f32 * 3)())
    for x, y in zip(_state(m), _state(fresh), strict=True):
        assert np.array_equal(x, y)


def test_a_fit_does_not_begin():
    rng = np.random.default_rng(1)
    x, t = (rng.standard_normal((64, 16)).astype(np.float32) for _ in range(2))
    net = Network(dims=(16, 32, 16))
    before = [w.copy() for pair in net.weights() for w in pair]
    net.status[:] = net.torch.tensor([_lib.ETIMEOUT, 7, 3], dtype=net.torch.int32)
    with pytest.raises(_lib.W2BError):
        net.fit(x, t, iters=4, batch=32)
    assert all(np.array_equal(a, w) for a, w in zip(before, (w for pair in net.weights() for w in pair), strict=True))
    net.status.zero_()
    assert len(net.fit(x, t, iters=4, batch=32)) == 2
