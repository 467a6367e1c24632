"""The flat FP32 step (yee_flat.cu) of grids whose rows are no multiple of four cells,
at the edges of its regions: CPMLs of one cell (no slab cell to update) and of all but
one row, plane counts that leave one, two or three planes to a thread, rows longer and
shorter than a block, conductivity, coefficients that differ on a cell's components.
Within 5e-5 of the restatement's peak, as the FP32 parity tests."""
from __future__ import annotations

import math

import numpy as np
import pytest

from bindings import OracleGrid


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,L", [
    (5, 6, 7, 1), (9, 10, 11, 3), (41, 14, 17, 6), (19, 271, 9, 2), (301, 12, 13, 4), (23, 17, 18, 5),
    (5, 4, 7, 0), (257, 5, 4, 0), (31, 33, 18, 0),
])
@pytest.mark.parametrize("one_coefficient", [True, False])
def test_flat_step_matches_restatement(fd, gpu, orc, nx, ny, nz, L, one_coefficient):
    dx = 0.05
    dt = 0.99 * dx / math.sqrt(3)
    rng = np.random.default_rng(nx + ny)
    grid = fd.Grid(nx, ny, nz, dx, fd.F32)
    g = OracleGrid(orc, nx, ny, nz, dx)
    ep = (1 + rng.integers(0, 3, (nz, ny, nx, 1 if one_coefficient else 3)) * 2.5) * np.ones(3)
    grid.ep[:] = ep.astype(np.float32)
    for m in range(3):
        g.ep[m][...] = ep[..., m]
    if L:
        fd.call("timefield3d_set_cpml", grid.t, L, 3, -1.0, 1.5, 0.05)
        g.set_boundary(orc.CPML)
        g.set_cpml(L, 3, -1.0, 1.5, 0.05, dt)
    else:
        fd.call("timefield3d_set_boundary", grid.t, fd.PEC)
        g.set_boundary(orc.PEC)
    fd.call("timefield3d_sync_device", grid.t)
    for n in range(12):
        v = float(np.float32(math.sin(0.7 * n + 0.3)))
        i, j, k = nx // 2, ny // 2, nz // 2
        fd.call("timefield3d_set_source_value", grid.t, i, j, k, 2, v)
        g.src[2][k, j, i] = v
        fd.call("timefield3d_apply_timestep_omp_full", grid.t, dt)
        g.step(dt)
    got, ref = grid.fields(), g.fields()
    peak = np.abs(ref).max()
    assert peak > 0
    assert np.abs(got - ref).max() <= 5e-5 * peak
    grid.close()
