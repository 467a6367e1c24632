"""Every family of bounded device waits runs out and says so: the self-test makes each
wait for what never comes (three launches: fused step, streaming tile, mode solver)
and reports FDTD_ERR_TIMEOUT only when all gave up."""
from __future__ import annotations

import ctypes as C

import pytest


@pytest.mark.gpu
def test_all_waits_give_up(fd, gpu):
    el = C.c_double()
    before = fd.lib.fdtd_launch_count()
    assert fd.lib.fdtd_wait_selftest(0.02, C.byref(el)) == fd.FDTD_ERR_TIMEOUT
    fd.lib.fdtd_clear_error()
    assert fd.lib.fdtd_launch_count() - before == 3
    assert 0.02 <= el.value < 1.0
    g = fd.Grid(16, 16, 16, 0.02, fd.F32)   # the context is in good order
    fd.call("timefield3d_set_cpml", g.t, 4, 3, -1.0, 1.0, 0.0)
    fd.lib.timefield3d_set_source_value(g.t, 8, 8, 8, 2, 1.0)
    fd.call("timefield3d_run", g.t, 0.01, 10)
    assert abs(g.fields()).max() > 0
    g.close()
