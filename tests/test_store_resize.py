"""An edge store whose buffers are made anew between two runs (used meanwhile on a grid of
another precision): the next run writes to the new ones, not through a graph captured
with the old addresses.  Read from the store: its second half equals an undisturbed
run's, its first half is gone with the old buffers."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import pytest

NX, NY, NZ, T = 40, 28, 40, 80


def grid(fd, precision):
    g = fd.Grid(NX, NY, NZ, 0.05, precision)
    fd.call("timefield3d_set_cpml", g.t, 6, 3, -1.0, 1.0, 0.0)
    fd.call("timefield3d_set_source_value", g.t, 20, 14, 20, 1, 1.0)
    return g


@pytest.mark.gpu
def test_run_after_the_store_was_remade(fd, gpu):
    dt = 0.99 * 0.05 / math.sqrt(3)
    left, right = (C.c_int * 2)(12, 12), (C.c_int * 2)(28, 28)
    out = []
    for disturb in (False, True):
        g, other = grid(fd, fd.F32), grid(fd, fd.F64)
        t = fd.call("adjoint3d_taper_new", 12.1, 1.0, 1, 15, 25, left, right, 10, 18, T)
        fd.call("adjoint3d_taper_bind_store", t, g.t, 0, 0, 1)
        fd.call("timefield3d_run", g.t, dt, 40)
        if disturb:
            for h in (other, g):
                fd.lib.adjoint3d_taper_store_forward_fields(t, h.t, 0)
                fd.check("store")
        fd.call("timefield3d_run", g.t, dt, 40)
        fd.call("adjoint3d_taper_sync_host", t)
        cells = 2 * 8 * 10
        f = np.ctypeslib.as_array(t.forward_fields, (T * cells * 6,)).reshape(T, cells * 6).copy()
        out.append(f)
        fd.call("adjoint3d_taper_unbind_store", t, g.t)
        fd.lib.adjoint3d_taper_free(t)
        g.close()
        other.close()
    assert np.abs(out[0][40:]).max() > 0 and np.abs(out[0][1:40]).max() > 0
    assert np.array_equal(out[0][40:], out[1][40:])
    assert np.abs(out[1][1:40]).max() == 0
