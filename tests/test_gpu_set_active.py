"""w2b_set_active alone decides which tiles a host-driven step takes: the per-tile flags follow the list, so a caller who
sets a list and then has the state arrays in hand gets the steps that the same list gives untouched."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from wadi2d_b200 import _lib
from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.model import Model
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu


def _model():
    import torch

    grid = TileGrid.from_mask(np.ones((60, 250), bool), 0.0, 0.0, 10.0)
    rng = np.random.default_rng(4)
    z = 0.3 * rng.random((grid.shape[0] * 2, grid.shape[1] * 2))
    m = Model(build_tables(grid, ArrayBed(z, 5.0), Tables(face_conveyance="strips")), Numerics())
    depth = np.zeros(grid.shape)
    depth[1:61, 1:90] = np.linspace(0.2, 0.9, 89)[None, :]
    m.set_depth(depth)
    b = m.backend
    b._t["is_act"].zero_()  # as the caller left them
    tiles = torch.as_tensor(np.arange(1, grid.ntiles - 3, dtype=np.int32), device=b.device)
    _lib.call("w2b_set_active", b.handle, tiles.data_ptr(), int(tiles.numel()), b._stream())
    return m, tiles


def test_flags_follow_the_list():
    m, tiles = _model()
    flags = np.zeros(m.grid.ntiles, np.int32)
    flags[tiles.cpu().numpy()] = 1
    assert np.array_equal(m.backend._t["is_act"].cpu().numpy(), flags)
    _lib.call("w2b_set_active", m.backend.handle, None, 0, m.backend._stream())
    assert not m.backend._t["is_act"].cpu().numpy().any()


@pytest.mark.parametrize("timed", [False, True], ids=["one_launch", "kernels"])
def test_fetching_the_state_changes_no_step(timed):
    def go(fetch: bool):
        m, _ = _model()
        b, p, ms = m.backend, ctypes.c_void_p(), (ctypes.c_float * 3)()
        for s in range(12):
            if fetch and s % 3 == 2:
                _lib.call("w2b_field_ptr", b.handle, _lib.FIELD_ID["h"], ctypes.byref(p))
            if timed:
                _lib.call("w2b_step_timed", b.handle, 0.3, int(s % 4 == 0), 0, b._stream(), ms)
            else:
                b.step(0.3, s % 4 == 0, False)
        return [b.get_field(f) for f in ("h", "d", "u", "v", "mx", "my", "qx", "qy", "res")]

    for a, b in zip(go(False), go(True), strict=True):
        assert np.array_equal(a, b)
