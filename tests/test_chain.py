"""timefield3d_run's chains of steps (the one-coefficient FP32 step, whose launches take
along the end of the step before) against the same steps by single calls, bit for bit:
fields, monitors, edge stores, the source plane with a value the schedule does not
touch.  Runs that end inside, at and after a graph's 32 steps, and are continued; no
store, two, and more than a chain takes."""
from __future__ import annotations

import ctypes as C
import math
import os

import numpy as np
import pytest

DP = C.POINTER(C.c_double)
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")
T = 150


def simulate(fd, nx, ny, nz, pieces, nmon, nstore):
    dx, L, src_z = 0.05, 6, 12
    dt = 0.99 * dx / math.sqrt(3)
    omega = 2 * fd.REF_PI / 1.55
    cx, cy = nx // 2, ny // 2
    g = fd.Grid(nx, ny, nz, dx, fd.F32)
    fd.lib.timefield3d_set_background(g.t, 2.085, 1.0)
    fd.lib.timefield3d_set_waveguide(g.t, 12.1, cx - 5, cx + 5, 0, nz, cy - 2, cy + 3)
    fd.call("timefield3d_set_cpml", g.t, L, 3, -1.0, 1.0, 0.0)
    m = fd.read_mode_file(os.path.join(GOLDEN, "modes", "small_te0.txt.gz"))
    om = np.array([omega * 0.97, omega, omega * 1.03])
    mons = [fd.call("timefield3d_add_overlap_monitor", g.t, cx, cy, z, m.copy().struct, 0, 3, om.ctypes.data_as(DP))
            for z in (16, nz - 14)[:nmon]]
    left, right = (C.c_int * 3)(cx - 6, cx - 7, cx - 8), (C.c_int * 3)(cx + 6, cx + 7, cx + 8)
    tapers = []
    for s in range(nstore):
        t = fd.call("adjoint3d_taper_new", 12.1, 1.0, 2, 18, 26, left, right, cy - 2, cy + 3 - s % 2, T)
        fd.call("adjoint3d_taper_bind_store", t, g.t, s % 2, T if s % 2 else 0, -1 if s % 2 else 1)
        tapers.append(t)
    # a value in the source's plane outside the mode's window: it stays
    fd.call("timefield3d_set_source_value", g.t, 8, ny - 5, src_z, 1, 0.25)
    amps = np.array([math.exp(-((n - 60) ** 2) / (2 * 20.0 ** 2)) for n in range(T)])
    phases = np.array([n * dt * omega for n in range(T)])
    if pieces:
        fd.call("timefield3d_set_source_schedule", g.t, cx, cy, src_z, m.struct, 0, 0, T, amps.ctypes.data_as(DP),
                phases.ctypes.data_as(DP))
        for n in pieces:
            fd.call("timefield3d_run", g.t, dt, n)
    else:
        for n in range(T):
            fd.lib.timefield3d_mode_source(g.t, cx, cy, src_z, m.struct, phases[n], amps[n], 0)
            fd.lib.timefield3d_apply_timestep_omp_full(g.t, dt)
        fd.check("stepwise")
    assert fd.lib.timefield3d_step_count(g.t) == T
    sums = []
    for mon in mons:
        acc = (fd.Complex * 3)()
        fd.call("timefield3d_read_overlap_monitor", g.t, mon, acc)
        sums.append([[a.re, a.im] for a in acc])
    stores = []
    for t in tapers:
        fd.call("adjoint3d_taper_sync_host", t)
        n = 6 * 2 * (t.top - t.bottom) * (t.end - t.start) * T
        stores += [np.ctypeslib.as_array(p, (n,)).copy() for p in (t.forward_fields, t.adjoint_fields)]
    f = g.fields()
    for t in tapers:
        fd.call("adjoint3d_taper_unbind_store", t, g.t)
        fd.lib.adjoint3d_taper_free(t)
    g.close()
    return f, np.array(sums), stores


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz", [(40, 28, 72), (64, 44, 40)])
@pytest.mark.parametrize("nmon,nstore", [(0, 0), (2, 0), (1, 2), (2, 5)])
def test_chains_equal_single_calls(fd, gpu, nx, ny, nz, nmon, nstore):
    f, sums, stores = simulate(fd, nx, ny, nz, None, nmon, nstore)
    assert np.abs(f).max() > 0 and (nmon == 0 or np.abs(sums).max() > 0)
    assert nstore == 0 or max(np.abs(s).max() for s in stores) > 0
    for pieces in ([T], [64, 86], [33, 1, 116]):
        f2, sums2, stores2 = simulate(fd, nx, ny, nz, pieces, nmon, nstore)
        assert np.array_equal(f, f2)
        assert np.array_equal(sums, sums2)
        assert all(np.array_equal(a, b) for a, b in zip(stores, stores2))
