"""Resident loops and fits on streams and threads of their own, more of them than fit the GPU together: each gives what it
gives alone, bit for bit, and none gives up waiting."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from wadi2d_b200.config import Numerics, Tables
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.model import Model
from wadi2d_b200.surrogate import Network
from wadi2d_b200.tables import ArrayBed, build_tables

pytestmark = pytest.mark.gpu
SIDES = ((62, 4), (126, 8), (62, 8), (254, 16), (62, 16), (126, 4), (254, 8), (62, 4))


def _model(side: int, rows: int):
    grid = TileGrid.from_mask(np.ones((side, side), bool), 0.0, 0.0, 10.0)
    z = 0.3 * np.random.default_rng(side + rows).random((grid.shape[0] * 2, grid.shape[1] * 2))
    m = Model(build_tables(grid, ArrayBed(z, 5.0), Tables(face_conveyance="strips")), Numerics())
    depth = np.zeros(grid.shape)
    depth[1 : side + 1, 1 : side + 1] = 0.4
    m.set_depth(depth)
    cfg = m.backend.loop_config()
    m.backend.set_loop(False, cfg[f"resident{rows}_occupancy"], 1, 32, strips=rows, resident=True)
    return m


def _step(m):
    for n in (20, 3, 33, 20, 20, 20):
        m.run(1e9, max_steps=n)
    for s in range(10):
        m.backend.step(0.2, s % 4 == 0, False)
    return [m.backend.get_field(f) for f in ("h", "u", "v", "qx", "res")] + [m.backend.max_wave()]


def _fit(seed: int):
    rng = np.random.default_rng(seed)
    x, t = (rng.standard_normal((300, 16)).astype(np.float32) for _ in range(2))
    net = Network(seed=seed)
    return [net.fit(x, t, iters=150, batch=256)] + [w for pair in net.weights() for w in pair]


def test_each_gives_what_it_gives_alone():
    import torch

    work = [lambda m=_model(*s): _step(m) for s in SIDES] + [lambda: _fit(1), lambda: _fit(2)]
    alone = [_step(_model(*s)) for s in SIDES] + [_fit(1), _fit(2)]
    torch.cuda.synchronize()
    got: list = [None] * len(work)
    go = threading.Barrier(len(work))

    def run(i: int) -> None:
        with torch.cuda.stream(torch.cuda.Stream()):
            go.wait()
            got[i] = work[i]()

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, got, strict=True):
        assert b is not None
        for x, y in zip(a, b, strict=True):
            assert np.array_equal(x, y)
