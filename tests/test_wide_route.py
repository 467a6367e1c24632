"""Grids with long rows and few cells: with a CPML the two-kernel step is the faster one
and FDTD_YEE_STREAM takes it, so its fields are FDTD_YEE_FLAT4's bit for bit; larger
grids go through tiles of the one-pass step, whose slab terms round differently; both
agree within the 5e-6 of the peak that the streaming step is held to."""
from __future__ import annotations

import numpy as np
import pytest

from test_tile_step import fields


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,nz,L,lossy,same", [(1000, 40, 40, 10, 0, True), (1900, 24, 20, 4, 1, True),
                                                   (1000, 70, 52, 3, 0, False)])
def test_route_of_grids_with_long_rows(fd, gpu, nx, ny, nz, L, lossy, same):
    a, b = (fields(fd, v, nx, ny, nz, L, lossy, 40, 0) for v in (fd.YEE_FLAT4, fd.YEE_STREAM))
    assert np.abs(a).max() > 0
    assert np.array_equal(a, b) == same
    assert np.abs(a - b).max() <= 5e-6 * np.abs(a).max()
