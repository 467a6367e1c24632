"""The tile plan of the one-coefficient streaming step (host computation): every quad of
the interior rows and planes belongs to one tile, tiles keep to what a block holds, and
no tile is a multiple of its share.

The last: a column's planes are cut into chunks of about equal time, a z-slab plane
counting 1.9, a y-slab band's plane up to twice an interior one's, and the chunks run
in at most two waves of blocks.  So a tile longer than 4 x 1.9 planes has at most
1.9 x 2 times the planes that an SM gets on average, and half a plane more at each end."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

NSM = 148
SHAPES = [(8, 5, 4, 0, 0), (12, 5, 30, 1, 0), (16, 16, 16, 4, 0), (24, 20, 18, 4, 1), (32, 32, 32, 6, 0),
          (48, 40, 44, 2, 0), (48, 40, 44, 6, 0), (48, 40, 44, 12, 0), (48, 40, 44, 0, 1), (64, 64, 64, 8, 0),
          (64, 64, 64, 10, 0), (64, 64, 64, 12, 0), (64, 48, 200, 8, 0), (96, 80, 64, 8, 1), (128, 72, 96, 10, 0),
          (128, 128, 128, 12, 0), (256, 128, 96, 12, 0), (200, 160, 400, 12, 0), (200, 160, 400, 0, 0),
          (384, 256, 384, 12, 0), (300, 300, 20, 6, 0), (1000, 40, 40, 10, 0), (1000, 40, 40, 6, 1), (64, 64, 1000, 10, 0),
          (512, 9, 300, 3, 0), (64, 500, 64, 10, 0)]


def plan(fd, nx, ny, nz, L, lossy, nsm=NSM):
    tp, th, sm = C.c_int(), C.c_int(), C.c_longlong()
    n = fd.lib.fdtd_tile_plan(nx, ny, nz, L, lossy, nsm, None, 0, C.byref(tp), C.byref(th), C.byref(sm))
    if n < 0:
        return None
    buf = (C.c_int * (6 * n))()
    assert fd.lib.fdtd_tile_plan(nx, ny, nz, L, lossy, nsm, buf, n, C.byref(tp), C.byref(th), C.byref(sm)) == n
    return np.array(buf, dtype=np.int64).reshape(n, 6), tp.value, th.value, sm.value


@pytest.mark.parametrize("shape", SHAPES)
def test_tiles_cover_the_interior_once(fd, shape):
    nx, ny, nz, L, lossy = shape
    tiles, tp, threads, smem = plan(fd, *shape)
    assert threads % 32 == 0 and threads <= 512 and smem <= 231424
    owned = np.zeros((nz, ny, nx // 4), dtype=np.int64)
    for q0, q1, j0, rows, k0, k1 in tiles:
        assert 0 <= q0 < q1 <= nx // 4 and 1 <= rows <= tp - 1 and 1 <= j0 and j0 + rows <= ny - 1
        assert 1 <= k0 < k1 <= nz - 1
        # a box of the tile's quads with its halo quads: 256 cells at most
        assert q1 - q0 + (q0 > 0) + (q1 < nx // 4) <= 64
        owned[k0:k1, j0:j0 + rows, q0:q1] += 1
    assert (owned[1:-1, 1:-1] == 1).all() and owned.sum() == (nz - 2) * (ny - 2) * (nx // 4)


@pytest.mark.parametrize("shape", SHAPES)
def test_no_tile_is_a_multiple_of_its_share(fd, shape):
    tiles = plan(fd, *shape)[0]
    columns = len({tuple(t[:4]) for t in tiles})
    share = columns * (shape[2] - 2) / NSM
    longest = max(k1 - k0 for *_, k0, k1 in tiles)
    assert longest <= max(4 * 1.9, 2 * 1.9 * share + 1)


def test_plan_rejects_what_the_step_does_not_take(fd):
    assert plan(fd, 30, 20, 20, 4, 0) is None     # rows of no whole quads
    assert plan(fd, 200, 160, 400, -1, 0) is None
    assert plan(fd, 200, 160, 400, 12, 0, 0) is None
