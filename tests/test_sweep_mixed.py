"""A candidate sweep whose grids take both routes of fdtd_sweep_run: one with equal E
coefficients on every cell's components (its own stream) and two with a cell where
they differ (the persistent launches).  Each ends as when run alone, bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_sweep import make_grid, monitors


def grid(fd, nz, T, differs):
    g, mons, dt = make_grid(fd, nz, T, "cpml", False)
    if differs:
        g.ep[nz // 2, 20, 24, 1] += 0.5
        fd.call("timefield3d_upload_materials", g.t)
    return g, mons, dt


@pytest.mark.gpu
def test_sweep_of_both_kinds_equals_single_runs(fd, gpu):
    kinds, steps = ((44, True), (60, False), (52, True)), (150, 97, 71)
    alone = []
    for (nz, differs), n in zip(kinds, steps):
        g, mons, dt = grid(fd, nz, 200, differs)
        fd.call("timefield3d_run", g.t, dt, n)
        alone.append((g.fields(), monitors(fd, g, mons), fd.lib.timefield3d_step_count(g.t)))
        g.close()
    grids = [grid(fd, nz, 200, differs) for nz, differs in kinds]
    arr = (fd.Timefield3d * 3)(*[g.t for g, _, _ in grids])
    fd.call("fdtd_sweep_run", arr, 3, grids[0][2], (C.c_int * 3)(*steps), 64, 0, 1.0)
    for (g, mons, _), (f, m, count) in zip(grids, alone):
        assert fd.lib.timefield3d_step_count(g.t) == count
        assert np.abs(m).max() > 0
        assert np.array_equal(monitors(fd, g, mons), m)
        assert np.array_equal(g.fields(), f)
        g.close()
