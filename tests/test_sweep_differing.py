"""The persistent launches (yee_sweep.cu) on what they are left with, grids whose
coefficients differ on a cell's components: CPML and PEC walls, with and without
conductivity, uneven step counts, and a second sweep that continues the first.  Each
grid ends as when run alone, bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_sweep import make_grid, monitors


def grid(fd, nz, T, boundary, lossy):
    g, mons, dt = make_grid(fd, nz, T, boundary, lossy)
    g.ep[nz // 2, 20, 24, 1] += 0.5
    fd.call("timefield3d_upload_materials", g.t)
    return g, mons, dt


@pytest.mark.gpu
@pytest.mark.parametrize("boundary", ["cpml", "pec"])
@pytest.mark.parametrize("lossy", [False, True])
def test_persistent_sweep_equals_single_runs(fd, gpu, boundary, lossy):
    nzs, first, second = (44, 60, 76), (150, 97, 203), (40, 71, 0)
    T, alone = 400, []
    for nz, a, b in zip(nzs, first, second):
        g, mons, dt = grid(fd, nz, T, boundary, lossy)
        fd.call("timefield3d_run", g.t, dt, a)
        if b:
            fd.call("timefield3d_run", g.t, dt, b)
        alone.append((g.fields(), monitors(fd, g, mons), fd.lib.timefield3d_step_count(g.t)))
        g.close()
    grids = [grid(fd, nz, T, boundary, lossy) for nz in nzs]
    arr = (fd.Timefield3d * 3)(*[g.t for g, _, _ in grids])
    for steps in (first, second):
        fd.call("fdtd_sweep_run", arr, 3, grids[0][2], (C.c_int * 3)(*steps), 64, 0, 1.0)
    for (g, mons, _), (f, m, count) in zip(grids, alone):
        assert fd.lib.timefield3d_step_count(g.t) == count
        assert np.abs(m).max() > 0
        assert np.array_equal(monitors(fd, g, mons), m)
        assert np.array_equal(g.fields(), f)
        g.close()
