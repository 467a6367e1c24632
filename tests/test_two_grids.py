"""Grids of different size and boundary alive at once, stepped in turn: the streaming
kernels' shared-memory limit is the process's, so preparing a grid whose tiles need
less must not take it from one whose tiles need more.  Each ends as when run alone,
bit for bit; `one_cell` makes a cell's coefficients differ (yee_stream.cu instead of
yee_tile.cu).  Bytes a block, 148 SMs, yee_tile.cu: 219488 for the first grid, 216032,
207392 for the next two."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

SHAPES = [(144, 75, 24, 6), (256, 40, 24, 6), (200, 60, 20, 0)]


def make(fd, nx, ny, nz, L, one_cell):
    dx = 0.05
    g = fd.Grid(nx, ny, nz, dx, fd.F32)
    rng = np.random.default_rng(nx)
    g.ep[:] = np.repeat((1 + rng.integers(0, 3, (nz, ny, nx, 1)) * 2.5), 3, axis=-1).astype(np.float32)
    if one_cell:
        g.ep[nz // 2, ny // 2, nx // 2, 1] += 1
    if L:
        fd.call("timefield3d_set_cpml", g.t, L, 3, -1.0, 1.5, 0.05)
    else:
        fd.call("timefield3d_set_boundary", g.t, fd.PEC)
    fd.call("timefield3d_set_yee_variant", g.t, fd.YEE_STREAM)
    fd.call("timefield3d_sync_device", g.t)
    for q in range(24):
        fd.lib.timefield3d_set_source_value(g.t, 7 + 3 * q, 9 + q, nz // 2, q % 6, float(rng.normal()))
    return g, 0.99 * dx / math.sqrt(3)


@pytest.mark.gpu
@pytest.mark.parametrize("one_cell", [0, 1])
def test_grids_in_turn_equal_grids_alone(fd, gpu, one_cell):
    turns = [("step", 1), ("run", 40), ("step", 2), ("run", 33)]

    def go(g, dt, what, n):
        if what == "run":
            fd.call("timefield3d_run", g.t, dt, n)
        else:
            for _ in range(n):
                fd.call("timefield3d_apply_timestep_omp_full", g.t, dt)

    alone = []
    for shape in SHAPES:
        g, dt = make(fd, *shape, one_cell)
        for t in turns:
            go(g, dt, *t)
        alone.append(g.fields())
        g.close()
    grids = [make(fd, *shape, one_cell) for shape in SHAPES]
    for t in turns:
        for g, dt in grids:
            go(g, dt, *t)
    for (g, _), f in zip(grids, alone):
        assert np.abs(f).max() > 0
        assert np.array_equal(g.fields(), f)
        g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("one_cell", [0, 1])
def test_sweep_of_grids_that_differ_in_rows_and_columns(fd, gpu, one_cell):
    shapes, steps = [SHAPES[0], (96, 44, 20, 6), SHAPES[1]], (45, 70, 33)
    alone = []
    for shape, n in zip(shapes, steps):
        g, dt = make(fd, *shape, one_cell)
        fd.call("timefield3d_run", g.t, dt, n)
        alone.append(g.fields())
        g.close()
    grids = [make(fd, *shape, one_cell) for shape in shapes]
    arr = (fd.Timefield3d * 3)(*[g.t for g, _ in grids])
    for half in range(2):   # continued: the same grids again, in the order of their preparation
        part = [n // 2 if half == 0 else n - n // 2 for n in steps]
        fd.call("fdtd_sweep_run", arr, 3, grids[0][1], (C.c_int * 3)(*part), 64, 0, 2.0)
    for (g, _), f in zip(grids, alone):
        assert np.abs(f).max() > 0
        assert np.array_equal(g.fields(), f)
        g.close()
