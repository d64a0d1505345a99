"""The work a program has this framework do, as cases that can be timed and compared: the time step in its device loop
(small, ordinary, ragged and the largest grids; every tile stepped or dry tiles asleep; both arithmetics), in the host
loop, in a run driver's window and in batches of runs, the table build, and the surrogate network's training and
prediction. Sizes are those of the configurations of ``wadi2d_b200.workloads`` and ``bench.py``, whole or reduced.

Every input is made from the case's seed on the GPU. ``prepare`` leaves a model as a run finds it: tables built, launch
schedule settled, wet start, rain falling. ``run`` is one pass through the public calls. ``exact`` computes the same
outputs in 64 bits with plain torch, from the tables, state and settings that the pass starts from.
"""

from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from wadi2d_b200.backend import BoundaryCells
from wadi2d_b200.batch import Batch
from wadi2d_b200.config import G, Numerics, Tables
from wadi2d_b200.forcing import ScsCurveNumber, UniformStorm
from wadi2d_b200.grid import TileGrid
from wadi2d_b200.maxima import Maxima, Tally
from wadi2d_b200.model import Model
from wadi2d_b200.run import DeviceRain, DeviceStorage, run_windows
from wadi2d_b200.state import state_index
from wadi2d_b200.surrogate import DIMS, Network
from wadi2d_b200.tables import ArrayBed, CrestFaces, build_tables

DEV = "cuda"
F64 = torch.float64

# What a step cannot do without, a cell (state read 44 B and written 40 B, static scalars 60 B, table values 40 B),
# with the envelope's share at every fourth step 10 B; and about the operations of its two faces and its update.
STEP_BYTES, STEP_FLOPS = 194, 420


# ------------------------------------------------------------------------------------------------ the cases


def listed() -> list[dict]:
    plane = {"bed": "plane", "dx": 10.0, "k": 5, "arith": "exact"}
    return [
        # configuration 1 at the size the unit studies and quick checks run it: launches and latency are all of it
        {"name": "loop_62", "kind": "loop", "ny": 62, "nx": 62, "steps": 20, "asleep": True, **plane},
        # configuration 1 whole: 256 x 256, the reference's arithmetic, about a window of 30 s
        {"name": "loop_256", "kind": "loop", "ny": 256, "nx": 256, "steps": 20, "asleep": True, **plane},
        # a flood in a valley with breaklines and Manning patches (configuration 2 reduced): most tiles asleep
        {"name": "loop_valley_1000x600", "kind": "loop", "bed": "valley", "ny": 1000, "nx": 600, "dx": 10.0, "k": 4,
         "arith": "exact", "steps": 20, "asleep": True},
        # an ordinary catchment, ragged sides, all wet, the reference's arithmetic
        {"name": "loop_1500x1101", "kind": "loop", "bed": "hills", "ny": 1500, "nx": 1101, "dx": 30.0, "k": 4,
         "arith": "exact", "steps": 13, "asleep": False},
        # configuration 3 whole: 4096 x 4096 at 30 m, the fast build, the 13 steps of a 30 s window
        {"name": "loop_4096", "kind": "loop", "bed": "hills", "ny": 4096, "nx": 4096, "dx": 30.0, "k": 4,
         "arith": "fast", "steps": 13, "asleep": False},
        # the host-driven loop that a run with callbacks, kicks or wake rules takes
        {"name": "host_256", "kind": "host", "ny": 256, "nx": 256, "seconds": 30.0, **plane},
        # the run driver's window on configuration 1: device rain with SCS loss, the steps, storage and books
        {"name": "window_256", "kind": "window", "ny": 256, "nx": 256, "seconds": 30.0, **plane},
        # the storm sweep (the critical-duration search): many storms on one catchment, tables shared
        {"name": "batch_shared_24x126", "kind": "batch", "bed": "hills", "runs": 24, "low": 126, "high": 126, "dx": 10.0,
         "k": 4, "arith": "exact", "shared": True, "steps": 20},
        # the ensemble (configuration 4 reduced): catchments of uneven size, each its own tables and cell size
        {"name": "batch_own_10x500", "kind": "batch", "bed": "hills", "runs": 10, "low": 90, "high": 500, "dx": 15.0,
         "k": 4, "arith": "fast", "shared": False, "steps": 13},
        # the table build: configuration 3's pixels (4 x 4 a cell, 7.5 m) and configuration 2's (10 x 10, 1 m) with
        # breaklines, local hydraulic radius as both have it
        {"name": "tables_1000", "kind": "tables", "bed": "hills", "ny": 1000, "nx": 1000, "dx": 30.0, "k": 4},
        {"name": "tables_1m_190x250", "kind": "tables", "bed": "valley", "ny": 190, "nx": 250, "dx": 10.0, "k": 10},
        # the surrogate of the screened search: 200 Adam steps at its batch of 256, then every candidate ranked
        {"name": "train_200", "kind": "train", "rows": 512, "batch": 256, "iters": 200, "predict": 2000},
    ]


def draw(rng) -> dict:
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["loop", "loop", "loop", "host", "window", "batch", "tables", "train"])
    if kind == "loop":
        bed = rng.choice(["plane", "hills", "hills", "valley"])
        top = {"plane": 1000, "hills": 2600, "valley": 1000}[bed]
        ny = side(40, top)
        nx = max(33, min(top, int(ny * math.exp(rng.uniform(-0.6, 0.6)))))
        return {"kind": kind, "bed": bed, "ny": ny, "nx": nx, "dx": 30.0 if bed == "hills" else 10.0,
                "k": rng.choice([4, 5]), "arith": rng.choice(["exact", "fast"]), "steps": rng.randint(8, 24),
                "asleep": bed == "valley" or rng.random() < 0.5}  # fmt: skip
    if kind in ("host", "window"):
        ny = side(60, 700)
        return {"kind": kind, "bed": "plane", "ny": ny, "nx": max(33, ny + rng.randint(-30, 30)), "dx": 10.0, "k": 5,
                "arith": "exact", "seconds": 30.0}  # fmt: skip
    if kind == "batch":
        shared = rng.random() < 0.5
        low = side(60, 250)
        return {"kind": kind, "bed": "hills", "runs": side(3, 40) if shared else rng.randint(2, 10), "low": low,
                "high": low if shared else side(low, 520), "dx": rng.choice([10.0, 15.0, 22.5]), "k": 4,
                "arith": rng.choice(["exact", "fast"]), "shared": shared, "steps": rng.randint(8, 24)}  # fmt: skip
    if kind == "tables":
        if rng.random() < 0.5:
            return {"kind": kind, "bed": "hills", "ny": side(60, 1000), "nx": side(60, 1000), "dx": 30.0,
                    "k": rng.choice([3, 4, 5, 6])}  # fmt: skip
        return {"kind": kind, "bed": "valley", "ny": side(40, 200), "nx": side(40, 250), "dx": 10.0,
                "k": rng.choice([5, 8, 10])}  # fmt: skip
    batch = rng.randint(48, 256)
    return {"kind": kind, "rows": batch + rng.randint(0, 300), "batch": batch, "iters": rng.randint(60, 250),
            "predict": side(100, 4000)}  # fmt: skip


# ------------------------------------------------------------------------------------------------ inputs


def _fractal(shape, gen):
    """A fractional Brownian surface (Hurst 0.8) of unit deviation, by spectral synthesis on the GPU."""
    white = torch.randn(shape, generator=gen, device=DEV)
    ky = torch.fft.fftfreq(shape[0], device=DEV)[:, None]
    kx = torch.fft.rfftfreq(shape[1], device=DEV)[None, :]
    kk = ky * ky + kx * kx
    kk[0, 0] = 1.0
    f = torch.fft.irfft2(torch.fft.rfft2(white).mul_(kk ** (-0.9)), s=shape)
    f -= f.mean()
    return f / f.std()


def _pad(n: int) -> int:
    return 32 * int(math.ceil((n + 2) / 32))


def _bed(case, ny, nx, dx, seed):
    """The pixels of a case's ground (FP64, on the GPU), Manning n and crest faces, on the padded grid."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    k, py, px = case["k"], _pad(ny), _pad(nx)
    x = (torch.arange(px * k, device=DEV, dtype=F64) + 0.5) * (dx / k) - dx
    y = (torch.arange(py * k, device=DEV, dtype=F64) + 0.5) * (dx / k) - dx
    fine = _fractal((py * k, px * k), g).double()
    manning, crest = 0.035, None
    if case["bed"] == "plane":  # configuration 1: 1 % eastward, a V-channel down the middle, 0.3 m of noise
        z = 100.0 + 0.01 * (nx * dx - x)[None, :] - 1.5 * torch.clamp(1 - (y - 0.5 * ny * dx).abs() / 20, min=0)[:, None]
        z = z + 0.3 * fine
    elif case["bed"] == "hills":  # configuration 3: relief falling south, 1.5 m of relief inside the cells
        relief = 0.012 * ny * dx
        coarse = _fractal((py, px), g).double()
        broad = F.interpolate(coarse[None, None], size=(py * k, px * k), mode="bilinear", align_corners=False)[0, 0]
        z = relief * (1.0 - y / (ny * dx))[:, None] + 0.06 * relief * broad + 1.5 * fine
    else:  # configuration 2: a valley falling south, a meandering channel, breaklines, Manning patches
        L, B = ny * dx, nx * dx
        c = 0.5 * B + 0.08 * B * torch.sin(2 * math.pi * y / (0.4 * L))
        off = (x[None, :] - c[:, None]).abs()
        z = 0.004 * (L - y)[:, None] + 30.0 * (off / B) ** 1.5 + 0.8 * fine
        z = z - 4.0 * torch.clamp(1 - off / 60.0, min=0.0)
        rng = np.random.default_rng(int(seed))
        manning = np.repeat(np.repeat(rng.choice([0.03, 0.04, 0.05, 0.06], (py // 32, px // 32)), 32, 0), 32, 1)
        crest = CrestFaces.empty((py, px))
        top = z.view(py, k, px, k).amax((1, 3)).cpu().numpy()
        for _ in range(40):  # levees along rows and columns, 0.5 - 3 m above the ground beside them
            j, i, n = int(rng.integers(2, ny - 1)), int(rng.integers(2, nx - 1)), int(rng.integers(10, 60))
            rise = rng.uniform(0.5, 3.0)
            if rng.random() < 0.5:
                jj = np.arange(j, min(j + n, ny))
                crest.xz[jj, i] = np.maximum(top[jj, i], top[jj, i - 1]) + rise
            else:
                ii = np.arange(i, min(i + n, nx))
                crest.yz[j, ii] = np.maximum(top[j, ii], top[j - 1, ii]) + rise
    return z, manning, crest


def _tables(case, ny, nx, dx, seed):
    z, manning, crest = _bed(case, ny, nx, dx, seed)
    grid = TileGrid.from_mask(np.ones((ny, nx), bool), 0.0, 0.0, dx)
    return build_tables(grid, ArrayBed(z, dx / case["k"]), Tables(), manning, crest=crest)


def _dense(grid, a):
    """A tile-layout tensor on the (ny, nx) grid, zero where no tile is."""
    ny, nx = grid.shape
    out = torch.zeros((ny // 32, nx // 32, 32, 32) + tuple(a.shape[3:]), dtype=a.dtype, device=a.device)
    t = torch.as_tensor(grid.tiles[1:].astype(np.int64), device=a.device)
    out[t[:, 0], t[:, 1]] = a[1:]
    return out.transpose(1, 2).reshape((ny, nx) + tuple(a.shape[3:]))


def _tab(tables, name):
    a = tables.device_arrays[name]
    return a if a.dim() > 2 else a.view((-1, 32, 32))


def _own(grid, native):
    """The (ny, nx) window of a NATIVE array (4 guard rows and 32 guard columns around the grid)."""
    ny, nx = grid.shape
    return native.view(ny + 8, nx + 64)[4 : 4 + ny, 32 : 32 + nx]


def _wet_start(case, tables, seed):
    """The mean depth that a pass starts from: 5 cm of water, more or less of it from place to place (the benchmark's
    wet start), or in the valley a flood that fills its channel up to 1.5 m and leaves the sides dry."""
    grid = tables.grid
    ny, nx = grid.shape
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 77)
    rough = torch.randn((ny // 8, nx // 8), generator=g, device=DEV)[None, None]
    rough = F.interpolate(rough, size=(ny, nx), mode="bilinear", align_corners=False)[0, 0].double()
    mask = torch.as_tensor(grid.mask, device=DEV)
    if case["bed"] != "valley":
        h = 0.05 * torch.exp(0.4 * rough)
    else:
        jj, ii = torch.nonzero(mask, as_tuple=True)
        n, m = int(jj.max()), int(ii.max())
        y = torch.arange(ny, device=DEV, dtype=F64)[:, None] / n
        c = m * (0.5 + 0.08 * torch.sin(2 * math.pi * y / 0.4))
        off = (torch.arange(nx, device=DEV, dtype=F64)[None, :] - c).abs() * grid.dx
        h = torch.clamp(1.5 - off / 60.0, min=0.0) * torch.exp(0.1 * rough) * (y < 0.6)
    return torch.where(mask, h, torch.zeros_like(h)).float()


def _rain(case, grid):
    """Rain excess, m/s: the configurations' 50 mm/h; in the valley a lumped inflow at the channel's head."""
    src = torch.zeros(grid.shape, device=DEV)
    mask = torch.as_tensor(grid.mask, device=DEV)
    if case["bed"] != "valley":
        return torch.where(mask, torch.full_like(src, 50.0 / 3.6e6), src)
    ny, nx = grid.shape
    src[1:3, nx // 2 - 2 : nx // 2 + 2] = 200.0 / (8 * grid.dx**2)
    return torch.where(mask, src, torch.zeros_like(src))


def _outlet(grid, bed):
    """Free-outfall cells: the east edge of the plane, a stretch of the south edge else."""
    jj, ii = np.nonzero(grid.mask)
    n, m = int(jj.max()), int(ii.max())
    if bed == "plane":
        return np.arange(1, n + 1), np.full(n, m)
    half = max(4, m // 16)
    cols = np.arange(max(1, m // 2 - half), min(m, m // 2 + half) + 1)
    return np.full(cols.size, n), cols


def _free(cells):
    n = cells.size
    zero = np.zeros(n, np.float32)
    return BoundaryCells(cells.astype(np.int32), cells.astype(np.int32), np.ones(n, np.int32), zero, zero)


FIELDS = ("h", "d", "u", "v", "qx", "qy")


def _put(backend, grid, h, tables, src, at=None):
    """The start of a run into the state arrays: mean depth h, its level and wet share, still water, the source."""
    for name in FIELDS + ("mx", "my", "res"):
        a = backend.native(name)
        (a if at is None else _own(grid, a)[at]).zero_()
    hc, dtab = _dense(tables.grid, _tab(tables, "hc")).double(), _dense(tables.grid, _tab(tables, "dtab"))
    d, om = _level(h.double(), hc, dtab)
    for name, v in (("h", h), ("d", d.float()), ("om", om.float()), ("src", src)):
        w = _own(grid, backend.native(name))
        (w if at is None else w[at]).copy_(v)


def _wet_tiles(grid, h):
    ny, nx = grid.shape
    blocks = (h > 0).view(ny // 32, 32, nx // 32, 32).any(3).any(1).cpu().numpy()
    wet = np.zeros(grid.ntiles, np.int32)
    wet[1:] = blocks[grid.tiles[1:, 0], grid.tiles[1:, 1]]
    return wet


def _settle(backend, advance):
    """Steps until the launch tuner has picked the loop's schedule, as a run's first second does."""
    for _ in range(64):
        if not backend.loop_config()["tuning"]:
            break
        advance()


def _model(case, seed):
    tables = _tables(case, case["ny"], case["nx"], case["dx"], seed)
    grid = tables.grid
    m = Model(tables, Numerics(arithmetic=case["arith"]))
    m.stepper.adaptive_active = bool(case.get("asleep", True))
    rows, cols = _outlet(grid, case["bed"])
    cells = np.asarray(state_index(grid, rows, cols), np.int64)
    m.set_boundary(_free(cells))
    h, src = _wet_start(case, tables, seed), _rain(case, grid)
    none = np.zeros(0, np.int64)
    x, y = (cells, none) if case["bed"] == "plane" else (none, cells)
    tally = Tally(m, x, np.ones(x.size), y, np.ones(y.size))
    kept = np.unique(np.concatenate((np.nonzero(_wet_tiles(grid, src))[0], m.boundary_tiles)))

    def start():
        """The model at the start of a run (the launch schedule, the graphs and the buffers stay)."""
        st = m.stepper
        _put(m.backend, grid, h, tables, src)
        m.backend.wet[:] = _wet_tiles(grid, h)
        st.t = 3600.0 if case["kind"] == "window" else 0.0  # an hour into the storm: the initial losses are met
        st.nsteps, st.dt, st.refresh_due = 0, st.num.cfl * grid.dx / st.num.wave_floor, True
        st.keep_active[:] = False
        st.keep_active[kept] = True
        st.rebuild_active()
        tally.total.zero_()
        return Maxima(m, 0.1, 0.05, every=4)

    maxima = start()
    if case["kind"] != "host":
        _settle(m.backend, lambda: m.run(1e12, maxima=maxima, tally=tally, max_steps=32))
        maxima = start()
    s = {"case": case, "model": m, "maxima": maxima, "tally": tally, "cells": (rows, cols)}
    if case["kind"] == "window":
        jj, ii = np.nonzero(grid.mask)
        every = np.asarray(state_index(grid, jj, ii), np.int64)
        cn = 60.0 + 30.0 * np.random.default_rng(int(seed)).random(every.size)
        s["cn"] = cn
        s["rain"] = DeviceRain(m, UniformStorm(2000.0, 2400.0), every, loss=ScsCurveNumber(cn))
        s["storage"] = DeviceStorage(m, every)
    torch.cuda.synchronize()
    return s


def _sides(case, seed):
    rng = np.random.default_rng(int(seed))
    n = case["runs"]
    lo, hi = math.log(case["low"]), math.log(case["high"])
    sides = np.round(np.exp(lo + (hi - lo) * (np.arange(n) + 0.5) / n)).astype(int)
    return [int(x) for x in sides], [float(np.round(case["dx"] * rng.uniform(0.8, 1.2), 2)) for _ in range(n)]


def _batch(case, seed):
    n = case["runs"]
    sides, dxs = _sides(case, seed)
    if case["shared"]:
        tabs = [_tables(case, sides[0], sides[0], case["dx"], seed)] * n
    else:
        tabs = [_tables(case, s, s, dx, seed + 1000 * r) for r, (s, dx) in enumerate(zip(sides, dxs, strict=True))]
    B = Batch([t.grid for t in tabs], tabs, Numerics(arithmetic=case["arith"]))
    cells = [_outlet(t.grid, case["bed"]) for t in tabs]
    ref = [np.asarray(state_index(t.grid, *c), np.int64) for t, c in zip(tabs, cells, strict=True)]
    B.set_boundary([_free(c) for c in ref])
    none = np.zeros(0, np.int64)
    B.set_tally([(none, none, c, np.ones(c.size)) for c in ref])
    at = [(slice(32 * p.oj, 32 * p.oj + t.grid.shape[0]), slice(32 * p.oi, 32 * p.oi + t.grid.shape[1]))
          for p, t in zip(B.place, tabs, strict=True)]  # fmt: skip
    grow = [0.5 + r / n for r in range(n)]  # every run a storm of its own
    src = [_rain(case, t.grid) * w for t, w in zip(tabs, grow, strict=True)]
    wet = [_wet_start(case, t, seed + 1000 * r) for r, t in enumerate(tabs)]

    def start():
        for r, t in enumerate(tabs):
            _put(B.backend, B.grid, wet[r], t, src[r], at[r])
        B.backend.wet[:] = 1
        B._pull()
        B.stepper.rebuild_active()
        B.set_source_tiles(np.arange(1, B.grid.ntiles))
        B.t[:], B.nsteps[:], B.refresh_due[:] = 0.0, 0, 1
        B.dt[:] = [B.num.cfl * float(t.grid.dx) / B.num.wave_floor for t in tabs]
        B.reset_envelope()
        B._tally.zero_()

    start()
    while True:  # whole rounds of an even number of steps leave every run on the same half of its pairs
        B.advance(1e12, max_every=4, max_steps=64)
        if not B.backend.loop_config()["tuning"]:
            break
    start()
    torch.cuda.synchronize()
    return {"case": case, "batch": B, "tables": tabs, "at": at, "cells": cells}


def _network(case, seed):
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    a = torch.randn((DIMS[0], DIMS[-1]), generator=g).numpy() / 4.0
    x = torch.randn((case["rows"], DIMS[0]), generator=g).numpy()
    t = np.tanh(x @ a) + 0.1 * x[:, :1] ** 2
    t = ((t - t.mean(0)) / t.std(0)).astype(np.float32)
    every = torch.randn((case["predict"], DIMS[0]), generator=g).numpy()
    return {"case": case, "net": Network(seed=int(seed) % 1000, lr=1e-4), "x": x, "t": t, "every": every}


def prepare(case: dict, seed: int) -> dict:
    if case["kind"] == "batch":
        return _batch(case, seed)
    if case["kind"] == "train":
        return _network(case, seed)
    if case["kind"] == "tables":
        z, manning, crest = _bed(case, case["ny"], case["nx"], case["dx"], seed)
        grid = TileGrid.from_mask(np.ones((case["ny"], case["nx"]), bool), 0.0, 0.0, case["dx"])
        return {"case": case, "grid": grid, "bed": ArrayBed(z, case["dx"] / case["k"]), "manning": manning,
                "crest": crest}  # fmt: skip
    return _model(case, seed)


# ------------------------------------------------------------------------------------------------ one pass


def _answer(backend, envelope, arith, tally):
    """The state after the pass and what it accumulated. What a threshold decides cell by cell (the speed and hazard
    where the water is over 5 cm, the arrival, the time of the first step over 10 cm) and the FP64 sums over float32
    discharges come back where the arithmetic is the reference's to the bit."""
    out = {name: backend.native(name) for name in FIELDS}
    out["max_depth"], out["max_mean_depth"] = envelope[0], envelope[1]
    if arith == "exact":
        out["max_speed"], out["max_hazard"], out["arrival"] = envelope[2:]
        if tally is not None:
            out["tally"] = tally
    return out


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "tables":
        return build_tables(state["grid"], state["bed"], Tables(), state["manning"],
                            crest=state["crest"]).device_arrays  # fmt: skip
    if kind == "train":
        net = state["net"]
        losses = net.fit(state["x"], state["t"], iters=case["iters"], batch=case["batch"], seed=1)
        return {"losses": losses, "W": net.W, "b": net.b, "predicted": net.forward(state["every"])}
    if kind == "batch":
        B = state["batch"]
        B.advance(1e12, max_every=4, max_steps=case["steps"])
        out = _answer(B.backend, B.backend.envelope(), case["arith"], B._tally)
        out["t"], out["dt"] = B.t, B.dt
        return out
    m, maxima, tally = state["model"], state["maxima"], state["tally"]
    st = m.stepper
    extra = {}
    if kind == "loop":
        m.run(1e12, maxima=maxima, tally=tally, max_steps=case["steps"])
    elif kind == "host":
        m.advance(st.t + case["seconds"], on_step=lambda s: maxima.update(s.t) if s.nsteps % 4 == 0 else None)
    else:
        done = run_windows(m, st.t + case["seconds"], rain=state["rain"], maxima=maxima, tally=tally,
                           storage=state["storage"])  # fmt: skip
        extra = {"rain": done.balance.rain, "storage": done.balance.storage}
    out = _answer(m.backend, maxima.arrays, case["arith"], None if kind == "host" else tally.total)
    return {**out, "t": st.t, "dt": st.dt, **extra}


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "train":
        dims = list(zip(DIMS[:-1], DIMS[1:], strict=True))
        mac, weights = sum(a * b for a, b in dims), sum(a * b + b for a, b in dims)
        flops = 2 * mac * (3 * case["batch"] * case["iters"] + case["predict"])
        # the batch's rows, the activations and gradients between layers, and the weights with their two moments
        acts = case["batch"] * (sum(DIMS) * 2 * 2 + sum(DIMS[1:]) * 4)
        return {"bytes": case["iters"] * (acts + weights * 24) + case["predict"] * 4 * (DIMS[0] + DIMS[-1]), "flops": flops}
    if kind == "batch":
        cells = sum(_pad(s) ** 2 for s in _sides(case, 0)[0])
    else:
        cells = _pad(case["ny"]) * _pad(case["nx"])
    if kind == "tables":
        k, pixel = case["k"], case["dx"] / case["k"]
        line = k + 2 * math.ceil(9.0 * 8.0 / pixel)  # a face's line at the least table top, 8 m
        return {"bytes": cells * (8 * k * k + 6 * 8 + 4 * (16 + 64 + 15) + 32), "flops": cells * (2 * 16 * line * 12)}
    if kind in ("host", "window"):
        steps = case["seconds"] / (0.45 * case["dx"] / 3.0)
    else:
        steps = case["steps"]
    share = 0.3 if case["bed"] == "valley" else 1.0  # of the tiles awake
    return {"bytes": STEP_BYTES * cells * steps * share, "flops": STEP_FLOPS * cells * steps * share}


# ------------------------------------------------------------------------------------------------ in 64 bits


def _f32(x) -> float:
    return float(np.float32(x))


def _level(h, hc, dtab):
    """Level over the lowest pixel and wet share of mean depths h, through the cell tables."""
    last = dtab.shape[-1] - 1
    s = torch.sqrt(torch.where(hc > 0, h / torch.where(hc > 0, hc, torch.ones_like(hc)), torch.zeros_like(h))) * last
    r = s.floor().clamp(0, last - 1).long()
    lo = dtab.gather(-1, r[..., None])[..., 0].double()
    hi = dtab.gather(-1, r[..., None] + 1)[..., 0].double()
    full = h >= hc
    d = torch.where(full, dtab[..., last].double() + (h - hc), lo + (s - r) * (hi - lo))
    om = hc * (2 * r + 1) / last**2 / (hi - lo).clamp(min=1e-12)
    flat = hc <= 0
    return torch.where(flat, h, d), torch.where(flat | full, torch.ones_like(om), om)


class Run64:
    """A run's step in 64 bits on dense (ny, nx) arrays: the sub-grid shallow-water step with every numerics switch on
    (second-order momentum, sheet flow, dry faces mirrored, carried face depth)."""

    def __init__(self, tables, num, dx, state, src, cells):
        g = tables.grid
        self.num, self.dx, self.src, self.cells = num, _f32(dx), src.double(), cells
        self.hc, self.dtab = _dense(g, _tab(tables, "hc")).double(), _dense(g, _tab(tables, "dtab"))
        have = torch.zeros((g.ntiles, 32, 32), device=DEV)
        have[1:] = 1.0
        self.void = _dense(g, have) == 0
        self.st = {}
        for ax in "xy":
            for n in ("fl", "fr", "gl", "gr", "ef", "cw", "ftab"):
                a = _dense(g, _tab(tables, n + ax))
                a = a if n == "ftab" else a.double()
                if n in ("fl", "fr"):
                    a[self.void] = 1e9
                if n == "ef":
                    a[self.void] = 1.0
                self.st[n + ax] = a
            self.st["zc" + ax] = _dense(g, _tab(tables, "zc" + ax)).double()
        for name, a in state.items():
            setattr(self, name, a.double())
        self.om = _level(self.h, self.hc, self.dtab)[1]
        self.mx, self.my = torch.zeros_like(self.h), torch.zeros_like(self.h)
        self.res = torch.zeros_like(self.h)
        self.env = [torch.zeros_like(self.h) for _ in range(4)] + [torch.full_like(self.h, -1.0)]
        self.tally = None
        self.t, self.dt, self.nsteps, self.due = 0.0, num.cfl * dx / num.wave_floor, 0, True

    def _faces(self, ax, dt, wave):
        P, dx, st = self.num, self.dx, self.st
        e_wet, h_cfl, a_min = _f32(P.e_wet), _f32(P.h_cfl), _f32(P.plan_min)
        g = _f32(G)
        zero = torch.zeros((), dtype=F64, device=DEV)

        def at(a):
            """Reader of a around each cell: steps along the face's axis, then across it."""
            p = F.pad(a, (2, 2, 2, 2))
            ny, nx = a.shape

            def get(s=0, c=0):
                j, i = (c, s) if ax == "x" else (s, c)
                return p[2 + j : 2 + j + ny, 2 + i : 2 + i + nx]

            return get

        U, V = (self.u, self.v) if ax == "x" else (self.v, self.u)
        Q, R = (self.qx, self.qy) if ax == "x" else (self.qy, self.qx)
        D, H, W = at(self.d), at(self.h), at(self.om)
        U_, V_, Q_, R_ = at(U), at(V), at(Q), at(R)
        fl, fr, gl, gr, top, cw = (st[n + ax] for n in ("fl", "fr", "gl", "gr", "ef", "cw"))
        Z = at(st["zc" + ax])
        e_l, e_r = D(-1) - fl, D() - fr
        p_l, p_r = e_l.clamp(min=0), e_r.clamp(min=0)
        left = (U > 0) | ((U == 0) & (e_l >= e_r))
        pick = lambda a, b: torch.where(left, a, b)  # noqa: E731
        eup = pick(p_l, p_r)
        live = eup > e_wet
        dz = pick(Z(-1) - fl, Z() - fr)
        phi = ((eup - 2 * dz) / (2 * dz)).clamp(0, 1)
        e = torch.where((cw == 0) & (dz > 1e-6), eup - phi * dz, eup)
        e = torch.where(live, e, torch.ones_like(e))
        h_l, h_r = H(-1), H()
        hup = pick(h_l, h_r)
        # the drive, where the downstream side stands below the face
        g_u, g_d, h_d = pick(gl, gr), pick(gr, gl), pick(h_r, h_l)
        drop = (hup - g_u) - torch.maximum(h_d - g_d, 0.5 * (g_u - g_d))
        drive = torch.maximum(eup, torch.minimum(drop, (e_l - e_r).abs()))
        d_eta = torch.where(pick(p_r, p_l) <= 0, pick(-drive, drive), p_r - p_l)
        # momentum fluxes, minmod-limited upwind velocities
        mirror = lambda a, own: torch.where(a == 0, own, a)  # noqa: E731

        def ustar(c, up, down):
            a, b = c - up, down - c
            return c + 0.5 * torch.where(a * b <= 0, zero, torch.where(a.abs() < b.abs(), a, b))

        def flux(um, uf, up, umm, upp, ql, qr):
            pl, pr = ql > 0, qr > 0
            sl = ustar(torch.where(pl, um, uf), torch.where(pl, umm, up), torch.where(pl, uf, um))
            sr = ustar(torch.where(pr, uf, up), torch.where(pr, um, upp), torch.where(pr, up, uf))
            return qr * sr - ql * sl

        um, up = mirror(U_(-1), U), mirror(U_(1), U)
        fx = flux(um, U, up, mirror(U_(-2), um), mirror(U_(2), up), 0.5 * (Q_(-1) + Q), 0.5 * (Q + Q_(1)))
        us_, un_ = mirror(U_(0, -1), U), mirror(U_(0, 1), U)
        fx = fx + flux(us_, U, un_, mirror(U_(0, -2), us_), mirror(U_(0, 2), un_), 0.5 * (R_(-1) + R_()),
                       0.5 * (R_(-1, 1) + R_(0, 1)))  # fmt: skip
        abar = 0.5 * (h_l + h_r) * dx
        press = dt * g * d_eta / dx
        mom = self.mx if ax == "x" else self.my
        us = torch.where(abar > _f32(1e-6) * dx, (mom - dt * fx / dx) / abar.clamp(min=1e-30), U) - press
        vb = 0.25 * (V_(-1) + V + V_(-1, 1) + V_(0, 1))
        # the face table
        tab = st["ftab" + ax]
        m = tab.shape[-2] - 1
        above = e >= top
        r = (torch.sqrt(e / top) * m).floor().clamp(0, m - 1).long()
        r = torch.where(above, torch.full_like(r, m - 1), r)
        flat = tab.view(tab.shape[:-2] + (-1,))
        at_row = lambda i: flat.gather(-1, i[..., None])[..., 0].double()  # noqa: E731
        a0, t0, a1, t1 = at_row(2 * r), at_row(2 * r + 1), at_row(2 * r + 2), at_row(2 * r + 3)
        rd = r.double()
        e0, de = (rd / m) ** 2 * top, (((rd + 1) / m) ** 2 - (rd / m) ** 2) * top
        f = (e - e0) / de
        w = (a1 - a0) / de
        area = torch.where(above, a1 + w * (e - top), a0 + f * (a1 - a0))
        tt = torch.where(above, t1 * area / a1.clamp(min=1e-12), t0 + f * (t1 - t0))
        avol = hup * dx
        sub = torch.minimum(p_l, p_r) / torch.maximum(p_l, p_r).clamp(min=1e-300)
        alpha = sub**4
        rho = torch.where(avol < area, alpha + (1 - alpha) * avol / area, torch.ones_like(area))
        fric = area**2 / tt.clamp(min=1e-300).pow(10 / 3).clamp(min=1e-30)
        fric = torch.where(rho < 1, fric / rho.clamp(min=1e-300).pow(4 / 3).clamp(min=1e-12), fric)
        a = dt * g * fric
        un = 2 * us / (1 + torch.sqrt(1 + 4 * a * torch.sqrt(us**2 + vb**2)))
        un = un.clamp(-P.u_max, P.u_max)
        qn = area * rho * un
        # crest faces: no more than critical flow over the section
        cap = cw * area * torch.sqrt(area / w.clamp(min=1e-9))
        over = (cw != 0) & (qn.abs() > cap)
        qn = torch.where(over, torch.where(qn > 0, cap, -cap), qn)
        un = torch.where(over, qn / (area * rho).clamp(min=1e-12), un)
        un, qn = torch.where(live, un, zero), torch.where(live, qn, zero)
        top_wave = 0.0
        if wave:
            o_l, o_r = W(-1), W()
            plan = pick(o_l, o_r)
            plan = torch.where(pick(D(), D(-1)) > h_cfl, torch.minimum(plan, pick(o_r, o_l)), plan)
            c = torch.sqrt((g * area * rho / (plan.clamp(min=a_min) * dx)).clamp(min=0))
            c = un.abs() + torch.minimum(P.dt_every * (un - U).abs(), 2 * c) + c
            c = torch.where(live & (pick(D(-1), D()) > h_cfl), c, zero)
            top_wave = float(c.max())
        return un, qn, abar * un, top_wave

    def step(self, rest, maxima_every, axis):
        P, dx = self.num, self.dx
        refresh = self.due or self.nsteps % P.dt_every == 0
        self.due = False
        dt = min(self.dt, rest, P.dt_max)
        u, qx1, mx, wx = self._faces("x", dt, refresh)
        v, qy1, my, wy = self._faces("y", dt, refresh)
        area = dx * dx
        east = lambda a: F.pad(a, (0, 1))[:, 1:]  # noqa: E731
        west = lambda a, fill: F.pad(a, (1, 0), value=fill)[:, :-1]  # noqa: E731
        south = lambda a: F.pad(a, (0, 0, 0, 1))[1:]  # noqa: E731
        north = lambda a, fill: F.pad(a, (0, 0, 1, 0), value=fill)[:-1]  # noqa: E731
        out = (east(qx1).clamp(min=0) + (-qx1).clamp(min=0) + south(qy1).clamp(min=0) + (-qy1).clamp(min=0)) * dt
        have = self.h.clamp(min=0) * area
        r = torch.where(out > have, have / out.clamp(min=1e-300), torch.ones_like(out))
        self.qx = qx1 * torch.where(qx1 > 0, west(r, 1.0), r)
        self.qy = qy1 * torch.where(qy1 > 0, north(r, 1.0), r)
        inc = self.res + dt * self.src - dt * (east(self.qx) - self.qx + south(self.qy) - self.qy) / area
        total = self.h + inc
        h = total.clamp(min=0)
        self.res = torch.where(total > 0, inc - (total - self.h), torch.zeros_like(inc))
        d, om = _level(h, self.hc, self.dtab)
        for a in (h, d):
            a[self.void] = 0.0
            a[self.cells] = 0.0
        if refresh:
            self.om = om
        self.u, self.v, self.mx, self.my, self.h, self.d = u, v, mx, my, h, d
        q = {"x": self.qx, "y": self.qy}[axis][self.cells]
        self.tally = (0 if self.tally is None else self.tally) + dt * q
        self.t += dt
        self.nsteps += 1
        if refresh:
            self.dt = min(P.cfl * dx / max(wx, wy, P.wave_floor), P.dt_max)
        if self.nsteps % maxima_every == 0:
            E = self.env
            E[0], E[1] = torch.maximum(E[0], d), torch.maximum(E[1], h)
            sp = torch.hypot(0.5 * (u + east(u)), 0.5 * (v + south(v)))
            deep = d > _f32(0.05)
            E[2] = torch.where(deep, torch.maximum(E[2], sp), E[2])
            E[3] = torch.where(deep, torch.maximum(E[3], sp * d), E[3])
            E[4] = torch.where((E[4] < 0) & (d >= _f32(0.1)), torch.full_like(d, self.t), E[4])


def _tiles(grid, dense, void=0.0):
    """A dense (ny, nx, ...) tensor in tile layout, the void tile ``void``."""
    ny, nx = grid.shape
    t = torch.as_tensor(grid.tiles[1:].astype(np.int64), device=DEV)
    b = dense.reshape((ny // 32, 32, nx // 32, 32) + tuple(dense.shape[2:])).transpose(1, 2)
    out = torch.full((grid.ntiles, 32, 32) + tuple(dense.shape[2:]), void, dtype=dense.dtype, device=DEV)
    out[1:] = b[t[:, 0], t[:, 1]]
    return out


def _exact_run(case, seed):
    s = prepare(case, seed)
    m = s["model"]
    grid, b, num = m.grid, m.backend, m.num
    cells = tuple(torch.as_tensor(c, device=DEV) for c in s["cells"])
    state = {n: _own(grid, b.native(n)).clone() for n in FIELDS}
    src = _own(grid, b.native("src")).clone()
    extra = {}
    t0 = m.stepper.t
    if case["kind"] == "window":  # the SCS loss of one window of the storm: 2,000 mm in 2,400 minutes
        keep = (1000.0 / torch.as_tensor(s["cn"], device=DEV) - 10.0) * 25.4
        fallen = []
        for t in (t0, t0 + case["seconds"]):
            p = (2000.0 / 2400.0 * t / 60.0 - 0.2 * keep).clamp(min=0)
            fallen.append(p**2 / (p + keep))
        rate = (fallen[1] - fallen[0]) / (1000.0 * case["seconds"])
        src = torch.zeros(grid.shape, dtype=F64, device=DEV)
        src[torch.as_tensor(grid.mask, device=DEV)] = rate
        extra["rain"] = float(rate.sum()) * grid.dx**2 * case["seconds"]
    R = Run64(m.tables, num, grid.dx, state, src, cells)
    axis = "x" if case["bed"] == "plane" else "y"
    R.t = t0
    steps, t_end = case.get("steps", 1 << 30), t0 + case.get("seconds", 1e12)
    while R.nsteps < steps and R.t < t_end - 1e-9:
        R.step(t_end - R.t, 4, axis)
    out = {n: F.pad(getattr(R, n), (32, 32, 4, 4)).reshape(-1) for n in FIELDS}
    env = [_tiles(grid, a, -1.0 if n == 4 else 0.0).reshape(-1) for n, a in enumerate(R.env)]
    out["max_depth"], out["max_mean_depth"] = env[:2]
    if case["arith"] == "exact":
        out["max_speed"], out["max_hazard"], out["arrival"] = env[2:]
        if case["kind"] != "host":  # the host loop takes no tally
            out["tally"] = R.tally
    if case["kind"] == "window":
        extra["storage"] = float((R.h + R.res).sum()) * grid.dx**2
    return {**out, "t": R.t, "dt": R.dt, **extra}


def _exact_batch(case, seed):
    s = prepare(case, seed)
    B = s["batch"]
    grid, b = B.grid, B.backend
    state = {n: _own(grid, b.native(n)).double() for n in FIELDS}
    src = _own(grid, b.native("src"))
    env = [torch.full((grid.ntiles, 1024), -1.0 if n == 4 else 0.0, dtype=F64, device=DEV) for n in range(5)]
    tally, t, dt = [], [], []
    for r, (tab, at) in enumerate(zip(s["tables"], s["at"], strict=True)):
        cells = tuple(torch.as_tensor(c, device=DEV) for c in s["cells"][r])
        R = Run64(tab, B.num, tab.grid.dx, {n: a[at].clone() for n, a in state.items()}, src[at], cells)
        for _ in range(case["steps"]):
            R.step(1e12, 4, "y")
        for n in FIELDS:
            state[n][at] = getattr(R, n)
        to = torch.as_tensor(B.map[r][1:], device=DEV)
        for n in range(5):
            env[n][to] = _tiles(tab.grid, R.env[n]).view(-1, 1024)[1:]
        tally.append(R.tally)
        t.append(R.t)
        dt.append(R.dt)
    out = {n: F.pad(a, (32, 32, 4, 4)).reshape(-1) for n, a in state.items()}
    env = [e.reshape(-1) for e in env]
    out["max_depth"], out["max_mean_depth"] = env[:2]
    if case["arith"] == "exact":
        out["max_speed"], out["max_hazard"], out["arrival"] = env[2:]
        out["tally"] = torch.cat(tally)
    out["t"], out["dt"] = np.array(t), np.array(dt)
    return out


def _exact_train(case, seed):
    s = prepare(case, seed)
    net = s["net"]
    W = [w.double() for w in net.W]
    b = [x.double() for x in net.b]
    X, T = (torch.as_tensor(s[n], device=DEV).double() for n in ("x", "t"))
    rng = np.random.default_rng(1)
    draws = [rng.choice(X.shape[0], size=case["batch"], replace=False) for _ in range(case["iters"])]

    def forward(x):
        for i, (w, c) in enumerate(zip(W, b, strict=True)):
            x = x @ w.T + c
            x = x.clamp(min=0) if i < len(W) - 1 else x
        return x

    params = W + b
    mom = [[torch.zeros_like(p), torch.zeros_like(p)] for p in params]
    losses = []
    for it, rows in enumerate(draws):
        for p in params:
            p.requires_grad_(True)
        at = torch.as_tensor(rows, device=DEV)
        loss = ((forward(X[at]) - T[at]) ** 2).mean()
        grads = torch.autograd.grad(loss, params)
        size = net.lr * math.sqrt(1 - 0.999 ** (it + 1)) / (1 - 0.9 ** (it + 1))
        for n, (p, g) in enumerate(zip(params, grads, strict=True)):
            p.requires_grad_(False)
            mom[n][0].mul_(0.9).add_(0.1 * g)
            mom[n][1].mul_(0.999).add_(0.001 * g * g)
            p.sub_(size * mom[n][0] / (mom[n][1].sqrt() + 1e-8))
        if it % 100 == 0 or it == case["iters"] - 1:
            losses.append(float(loss))
    every = torch.as_tensor(s["every"], device=DEV).double()
    return {"losses": losses, "W": W, "b": b, "predicted": forward(every)}


def _exact_tables(case, seed):
    s = prepare(case, seed)
    grid, cfg, k = s["grid"], Tables(), case["k"]
    ny, nx = grid.shape
    dx, last = case["dx"], cfg.rows - 1
    pixel = dx / k
    z = s["bed"].z
    margin = min(math.ceil(cfg.local_radius_beta * cfg.face_depth_max / pixel), max(z.shape))
    x2 = (torch.arange(cfg.rows, device=DEV, dtype=F64) / last) ** 2
    out = {}
    # cells: the mean-depth curve of the sorted pixels
    cell = z.view(ny, k, nx, k).transpose(1, 2)
    p = cell.reshape(ny, nx, k * k).sort(-1).values
    n = k * k
    zmin = p[..., 0]
    p = p - zmin[..., None]
    mean = p.mean(-1)
    hc = p[..., -1] - mean
    count = torch.arange(1, n + 1, device=DEV, dtype=F64)
    filled = ((p * count - p.cumsum(-1)) / n).cummax(-1).values
    want = hc[..., None] * x2
    at = torch.searchsorted(filled, want.contiguous(), right=True).sub_(1).clamp_(0, n - 1)
    tab = p.gather(-1, at) + (want - filled.gather(-1, at)) * n / (at + 1)
    tab[..., last] = p[..., -1]
    flat = hc <= 1e-9
    tab[flat] = 0.0
    out["hc"], out["dtab"] = torch.where(flat, torch.zeros_like(hc), hc), tab
    mid = (k // 2,) if k % 2 else (k // 2 - 1, k // 2)
    for ax, lines in (("x", [cell[..., :, c].amin(-1) for c in mid]), ("y", [cell[..., c, :].amin(-1) for c in mid])):
        out["zc" + ax] = (sum(lines) / len(lines) - zmin).clamp(min=0)
    dense = {"zmin": zmin, "zbar": zmin + mean}
    # faces: the strips' areas, and the conveyance by the local hydraulic radius along the face's line
    nman = torch.full((ny, nx), float(s["manning"]), dtype=F64, device=DEV) if np.isscalar(s["manning"]) else (
        torch.as_tensor(s["manning"], device=DEV, dtype=F64))  # fmt: skip
    mask = torch.as_tensor(grid.mask, device=DEV)
    crest = s["crest"]
    for ax in "xy":
        zz = z if ax == "x" else z.T
        msk = mask if ax == "x" else mask.T
        nm = nman if ax == "x" else nman.T
        A, B = (ny, nx) if ax == "x" else (nx, ny)  # along the faces, across them
        edge = torch.maximum(zz[:, (torch.arange(B, device=DEV) * k - 1).clamp(min=0)], zz[:, ::k])
        rows = (torch.arange(A, device=DEV)[:, None] * k + torch.arange(-margin, k + margin, device=DEV)).clamp(0, A * k - 1)
        given = None
        if crest is not None:
            a = torch.as_tensor(crest.xz if ax == "x" else crest.yz, device=DEV)
            given = a if ax == "x" else a.T
        got = {n: [] for n in ("ftab", "ef", "zf")}
        step = max(1, (1 << 25) // (B * (k + 2 * margin)))
        for a0 in range(0, A, step):
            sel = slice(a0, min(A, a0 + step))
            ext = edge[rows[sel]].transpose(1, 2).reshape(-1, k + 2 * margin)  # (faces, line)
            c = None if given is None else given[sel].reshape(-1)
            ft, top, zf = _face64(ext, c, nm[sel].reshape(-1), k, margin, pixel, cfg, x2)
            shape = (-1, B)
            got["ftab"].append(ft.view(shape + ft.shape[1:]))
            got["ef"].append(top.view(shape))
            got["zf"].append(zf.view(shape))
        v = {n: torch.cat(a) for n, a in got.items()}
        zf = v["zf"]
        roll = lambda a: torch.roll(a, 1, 1)  # noqa: E731
        lo, bar = (dense[n] if ax == "x" else dense[n].T for n in ("zmin", "zbar"))
        opened = msk & roll(msk)
        closed = torch.full_like(zf, 1e9)
        zero = torch.zeros_like(zf)
        v["fl"], v["fr"] = torch.where(opened, zf - roll(lo), closed), torch.where(opened, zf - lo, closed)
        v["gl"], v["gr"] = torch.where(opened, zf - roll(bar), zero), torch.where(opened, zf - bar, zero)
        sharp = (v["gl"] > cfg.crest_tolerance) & (v["gr"] > cfg.crest_tolerance)
        v["cw"] = torch.where(sharp, torch.full_like(zf, 1.7046), zero)
        for name in ("ftab", "ef", "fl", "fr", "gl", "gr", "cw"):
            out[name + ax] = v[name] if ax == "x" else v[name].transpose(0, 1)
    tiles = {name: _tiles(grid, a, 1.0 if name in ("efx", "efy") else 0.0) for name, a in out.items()}
    held = torch.zeros((ny // 32, nx // 32), dtype=torch.bool, device=DEV)
    held[tuple(torch.as_tensor(grid.tiles[1:].astype(np.int64), device=DEV).T)] = True
    held = held.repeat_interleave(32, 0).repeat_interleave(32, 1)
    return {**tiles, **{name: torch.where(held, a, torch.zeros_like(a)) for name, a in dense.items()}}


def _face64(ext, crest, nman, k, margin, pixel, cfg, x2):
    """Table (faces, rows, 2), top and invert of faces whose lines of pixels are ``ext``."""
    n = ext.shape[1]
    prof = ext[:, margin : margin + k]
    natural = torch.ones(ext.shape[0], dtype=torch.bool, device=DEV) if crest is None else torch.isnan(crest)
    if crest is not None:
        prof = torch.where(natural[:, None], prof, torch.maximum(prof, crest[:, None]))
    zf = prof.amin(1)
    top = (prof.amax(1) - zf).clamp(max=cfg.face_depth_max).clamp(min=cfg.face_depth_min)
    line = (ext.amax(1) - zf).clamp(max=cfg.face_depth_max)
    top = torch.where(natural, torch.maximum(top, line), top)
    e = torch.ceil(cfg.local_radius_beta * top / pixel).clamp(max=margin)
    pos = torch.arange(n, device=DEV)
    valid = (pos >= margin - e[:, None]) & (pos < margin + k + e[:, None])
    rise = ext[:, 1:] - ext[:, :-1]
    seg = torch.sqrt(pixel**2 + rise**2)
    both = valid[:, 1:] & valid[:, :-1]
    first, final = (margin - e).long()[:, None], (margin + k + e - 1).long()[:, None]
    ids = torch.arange(margin, margin + k, device=DEV)
    out = torch.empty((ext.shape[0], x2.numel(), 2), dtype=F64, device=DEV)
    for r in range(x2.numel()):
        dep = (top * x2[r])[:, None] - (prof - zf[:, None])
        dep = dep.clamp(min=0)
        out[:, r, 0] = pixel * dep.sum(1)
        strips = (dep * dep.pow(2 / 3)).sum(1)
        d = torch.where(valid, ((zf + top * x2[r])[:, None] - ext).clamp(min=0), torch.zeros_like(ext))
        wet = d > 0
        wa, wb = wet[:, :-1] & both, wet[:, 1:] & both
        da, db = d[:, :-1], d[:, 1:]
        half = torch.full_like(seg, 0.5 * pixel)
        up = torch.where(rise > 0, (da / rise).clamp(max=1) * seg, half)
        down = torch.where(rise < 0, (db / -rise).clamp(max=1) * seg, half)
        per = torch.zeros_like(ext)
        per[:, :-1] += torch.where(wa & wb, 0.5 * seg, torch.where(wa, up, torch.zeros_like(seg)))
        per[:, 1:] += torch.where(wa & wb, 0.5 * seg, torch.where(wb, down, torch.zeros_like(seg)))
        for end in (first, final):
            per.scatter_add_(1, end, 0.5 * pixel * wet.gather(1, end).double())
        run_lo = torch.where(wet, torch.full_like(pos, -1), pos).cummax(1).values + 1
        run_hi = n - 1 - ((n - 1 - torch.where(wet, torch.full_like(pos, n), pos)).flip(1).cummax(1).values.flip(1) + 1)
        zero = torch.zeros((ext.shape[0], 1), dtype=F64, device=DEV)
        sums = [torch.cat((zero, a.cumsum(1)), 1) for a in (d, pos * d, per, pos * per)]
        di = d[:, ids]
        i = ids.double()
        w = (cfg.local_radius_beta * di / pixel).clamp(min=1e-9)
        lo = torch.maximum(torch.ceil(i - w).long(), run_lo[:, ids]).clamp(0, n)
        hi = torch.minimum(torch.floor(i + w).long(), run_hi[:, ids]).clamp(-1, n - 1)

        def tent(s0, s1):
            lo0, mid0, hi0 = s0.gather(1, lo), s0[:, ids + 1], s0.gather(1, hi + 1)
            lo1, mid1, hi1 = s1.gather(1, lo), s1[:, ids + 1], s1.gather(1, hi + 1)
            return ((1 - i / w) * (mid0 - lo0) + (mid1 - lo1) / w) + ((1 + i / w) * (hi0 - mid0) - (hi1 - mid1) / w)

        a_sum, p_sum = tent(sums[0], sums[1]), tent(sums[2], sums[3])
        radius = torch.where(p_sum > 0, pixel * a_sum / torch.where(p_sum > 0, p_sum, torch.ones_like(p_sum)), di)
        local = torch.where(di > 0, di * radius.clamp(min=0).pow(2 / 3), torch.zeros_like(di)).sum(1)
        out[:, r, 1] = (pixel / nman * torch.where(natural, local, strips)).pow(0.6)
    return out, top, zf


def exact(case: dict, seed: int):
    if case["kind"] == "tables":
        return _exact_tables(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "batch":
        return _exact_batch(case, seed)
    return _exact_run(case, seed)
