"""A tile plan that could not be replaced (a device allocation that fails while the
grid's conductivity changes) leaves no half of it behind: the same call works once the
allocation does, and so does going back, bit for bit as on a grid that met no failure."""
from __future__ import annotations

import math

import numpy as np
import pytest

NX, NY, NZ = 64, 44, 30


def make(fd, one_cell):
    dx = 0.05
    g = fd.Grid(NX, NY, NZ, dx, fd.F32)
    rng = np.random.default_rng(3)
    g.ep[:] = np.repeat((1 + rng.integers(0, 3, (NZ, NY, NX, 1)) * 2.5), 3, axis=-1).astype(np.float32)
    if one_cell:
        g.ep[NZ // 2, NY // 2, NX // 2, 1] += 1
    fd.call("timefield3d_set_cpml", g.t, 6, 3, -1.0, 1.5, 0.05)
    fd.call("timefield3d_set_yee_variant", g.t, fd.YEE_STREAM)
    fd.call("timefield3d_sync_device", g.t)
    for q in range(24):
        fd.lib.timefield3d_set_source_value(g.t, 7 + 2 * q, 9 + q, NZ // 2, q % 6, float(rng.normal()))
    return g, 0.99 * dx / math.sqrt(3)


def conductivity(fd, g, value):
    fd.lib.timefield3d_set_prism_electric_conductivity(g.t, value, 20, 40, 10, 30, 8, 20)


@pytest.mark.gpu
@pytest.mark.parametrize("one_cell", [0, 1])
@pytest.mark.parametrize("back", [False, True])
def test_failed_replan_leaves_the_grid_usable(fd, gpu, one_cell, back):
    out = []
    for fail in (False, True):
        g, dt = make(fd, one_cell)
        for value in (0.3, 0.0):   # both settings run once: their coefficient arrays exist from here on
            conductivity(fd, g, value)
            fd.call("timefield3d_run", g.t, dt, 33)
        conductivity(fd, g, 0.3)
        if fail:
            before = g.fields()
            fd.lib.fdtd_inject_allocation_failures(1)
            fd.lib.timefield3d_run(g.t, dt, 33)
            assert fd.lib.fdtd_last_error() == fd.FDTD_ERR_ALLOC
            fd.lib.fdtd_clear_error()
            fd.lib.fdtd_inject_allocation_failures(0)
            assert np.array_equal(g.fields(), before)
        if back:
            conductivity(fd, g, 0.0)
        fd.call("timefield3d_run", g.t, dt, 45)
        out.append(g.fields())
        g.close()
    assert np.abs(out[0]).max() > 0
    assert np.array_equal(out[0], out[1])
