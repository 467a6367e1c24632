"""The one-coefficient streaming step (yee_tile.cu) where its tiles can go wrong:
rows in one to three tiles, bands of one row, planes that all lie in slabs, one and
two waves of tiles, conductivity.  Against the two-kernel step (FDTD_YEE_FLAT4) on
the same grid, within the 5e-6 of the peak that the streaming step is held to; the
same for a grid in which one cell's coefficients differ (yee_stream.cu takes it)."""
from __future__ import annotations

import math

import numpy as np
import pytest


def fields(fd, variant, nx, ny, nz, L, lossy, steps, one_cell):
    dx = 0.05
    dt = 0.99 * dx / math.sqrt(3)
    rng = np.random.default_rng(nx * ny + nz)
    g = fd.Grid(nx, ny, nz, dx, fd.F32)
    ep = np.repeat((1 + rng.integers(0, 3, (nz, ny, nx, 1)) * 2.5), 3, axis=-1).astype(np.float32)
    if one_cell:
        ep[nz // 2, ny // 2, nx // 2, 1] += 1
    g.ep[:] = ep
    if lossy:
        fd.lib.timefield3d_set_prism_electric_conductivity(g.t, 0.3, 2, nx - 3, 1, ny - 1, 1, nz - 1)
    if L:
        fd.call("timefield3d_set_cpml", g.t, L, 3, -1.0, 1.5, 0.05)
    else:
        fd.call("timefield3d_set_boundary", g.t, fd.PEC)
    fd.call("timefield3d_set_yee_variant", g.t, variant)
    fd.call("timefield3d_sync_device", g.t)
    planes = sorted({1 + (nz - 3) * q // 3 for q in range(4)})   # a grid holds sources in four planes at most
    for q in range(96):
        i, j = (int(rng.integers(1, n - 1)) for n in (nx, ny))
        fd.lib.timefield3d_set_source_value(g.t, i, j, planes[q % len(planes)], q % 6, float(rng.normal()))
    fd.call("timefield3d_run", g.t, dt, steps)
    fd.call("timefield3d_apply_timestep_omp_full", g.t, dt)
    out = g.fields()
    g.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,L,lossy", [
    (8, 5, 4, 0, 0), (12, 5, 30, 1, 0), (40, 30, 11, 4, 0), (128, 9, 40, 3, 1), (36, 21, 30, 5, 0),
    (300, 18, 20, 6, 0), (300, 9, 24, 0, 1), (520, 14, 12, 4, 1), (520, 20, 16, 0, 0),
    (96, 80, 64, 8, 1), (256, 128, 64, 10, 0), (200, 150, 40, 0, 0),
])
@pytest.mark.parametrize("one_cell", [0, 1])
def test_tile_step_matches_two_kernel_step(fd, gpu, nx, ny, nz, L, lossy, one_cell):
    a, b = (fields(fd, v, nx, ny, nz, L, lossy, 45, one_cell) for v in (fd.YEE_FLAT4, fd.YEE_STREAM))
    assert np.abs(a).max() > 0
    assert np.abs(a - b).max() <= 5e-6 * np.abs(a).max()
