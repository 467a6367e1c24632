"""The per-cell FP64/FP32 step (yee_split.cu) where its launches split: grids as
small as their slabs allow, a 1-cell CPML (no updated cell in a slab), the Mur
step's E faces inside the H launch, probes recorded by the step's last launch or,
on the shell, after it.  FP64 equals the restatement bit for bit; FP32 within
5e-5 of its peak, as its parity tests."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

from bindings import OracleGrid

DP = C.POINTER(C.c_double)


@pytest.mark.gpu
@pytest.mark.parametrize("prec,nx,ny,nz,L",
                         [(p, *s, 0) for p in ("f64", "f32") for s in ((4, 4, 4), (5, 4, 7), (257, 5, 4), (31, 33, 18))]
                         + [("f64", *s) for s in ((5, 6, 7, 1), (8, 9, 10, 3), (40, 14, 16, 6), (19, 270, 9, 2))])
def test_step_matches_restatement(fd, gpu, orc, prec, nx, ny, nz, L):
    dx = 0.05
    dt = 0.99 * dx / math.sqrt(3)
    rng = np.random.default_rng(nx + ny)
    grid = fd.Grid(nx, ny, nz, dx, fd.F64 if prec == "f64" else fd.F32)
    g = OracleGrid(orc, nx, ny, nz, dx)
    ep = np.repeat((1 + rng.integers(0, 3, (nz, ny, nx, 1)) * 2.5), 3, axis=-1).astype(np.float32)
    grid.ep[:] = ep
    for m in range(3):
        g.ep[m][...] = ep[..., m]
    if L:
        fd.call("timefield3d_set_cpml", grid.t, L, 3, -1.0, 1.5, 0.05)
        g.set_boundary(orc.CPML)
        g.set_cpml(L, 3, -1.0, 1.5, 0.05, dt)
    fd.call("timefield3d_sync_device", grid.t)
    cells = [(1, 1, 1), (nx - 1, ny // 2, 1), (nx // 2, ny // 2, nz // 2)]
    pids = [fd.call("timefield3d_add_probe", grid.t, *c, m, 32) for c in cells[:: 1 if nx % 2 else 2] for m in (1, 4)]
    where = [(c, m) for c in cells[:: 1 if nx % 2 else 2] for m in (1, 4)]
    want = []
    for n in range(12):
        v = float(np.float32(math.sin(0.7 * n)))
        i, j, k = nx // 2, ny // 2, nz // 2
        fd.call("timefield3d_set_source_value", grid.t, i, j, k, 2, v)
        g.src[2][k, j, i] = v
        fd.call("timefield3d_apply_timestep_omp_full", grid.t, dt)
        g.step(dt)
        f = g.fields()
        want.append([f[c[2], c[1], c[0], m] for c, m in where])
    got, ref = grid.fields(), g.fields()
    seen = np.zeros((len(pids), 12))
    for q, pid in enumerate(pids):
        fd.call("timefield3d_read_probe", grid.t, pid, seen[q].ctypes.data_as(DP), 12)
    assert fd.lib.timefield3d_step_count(grid.t) == 12
    if prec == "f64":
        assert np.array_equal(got, ref)
        assert np.array_equal(seen, np.array(want).T)
    else:
        peak = np.abs(ref).max()
        assert np.abs(got - ref).max() <= 5e-5 * peak
        assert np.abs(seen - np.array(want).T).max() <= 5e-5 * peak
