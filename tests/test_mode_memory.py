"""The mode solver's device memory with a Krylov size whose Gram matrix does not fit
shared memory: one matrix for the grid, not one for every block.

Window 60 x 40, K = 256: basis 257 x 4800 x 16 B = 20 MB, Gram and H 1 MB each, the
rest below 4 MB; a Gram matrix for each of 148 blocks would be 155 MB.  The bound leaves
as much again for what the driver takes in its 2 MB pieces."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.mark.gpu
def test_krylov_scratch_is_one_gram_matrix(fd, gpu):
    omega, disc, mi, mj = 2 * fd.REF_PI / 1.55, 0.05, 60, 40
    ep = np.full((mj, mi, 3), 2.085, complex)
    ep[mj // 2 - 3:mj // 2 + 2, mi // 2 - 5:mi // 2 + 5] = 12.1

    def solve(K):
        m = fd.HostMode(np.zeros((mj, mi, 6)), disc, ep)
        C.CDLL(None).srand(3)
        return fd.call("fdtd_mode_solve_beta_squared", C.byref(m.struct), omega, 1e-6, None, 0, K, 2, 0)

    want = solve(20)    # kernels loaded, context grown
    torch.cuda.mem_get_info()
    lowest, done = [], threading.Event()

    def watch():
        while not done.is_set():
            lowest.append(torch.cuda.mem_get_info()[0])

    before = torch.cuda.mem_get_info()[0]
    t = threading.Thread(target=watch)
    t.start()
    try:
        got = solve(256)
    finally:
        done.set()
        t.join()
    assert abs(complex(got.re, got.im) - complex(want.re, want.im)) < 1e-4 * abs(complex(want.re, want.im))
    used = before - min(lowest)
    assert 16e6 < used < 52e6
