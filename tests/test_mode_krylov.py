"""The mode solver's Krylov kernel over the sizes its variants split at: 1, 2, 4
or any number of vector elements a thread, Krylov sizes on both sides of a warp
and of the shared-memory Gram matrix, both boundary conditions.

The solved mode must satisfy its eigenproblem: with the operator the library
exports (bit-exact to the reference's), |B h - beta^2 h| <= 1e-4 |beta^2 h| over
the interior.  The solver stops when n_eff moves by less than tol = 1e-9 a
restart; the residual then stays far below that bound on these well-separated
modes."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("mi,mj,K,conf", [(24, 16, 20, 2), (60, 40, 33, 2), (137, 138, 20, 1), (139, 140, 20, 2),
                                          (220, 180, 12, 2), (280, 276, 20, 2), (90, 70, 112, 2)])
def test_solved_mode_satisfies_its_equation(fd, gpu, mi, mj, K, conf):
    omega, disc = 2 * fd.REF_PI / 1.55, 0.05
    ep = np.full((mj, mi, 3), 2.085, complex)
    ep[mj // 2 - 3:mj // 2 + 2, mi // 2 - 5:mi // 2 + 5] = 12.1
    m = fd.HostMode(np.zeros((mj, mi, 6)), disc, ep)
    C.CDLL(None).srand(3)
    beta = fd.call("fdtd_mode_solve_beta_squared", C.byref(m.struct), omega, 1e-9, None, 0, K, conf, 0)
    out = fd.HostMode(np.zeros((mj, mi, 6)), disc)
    fd.call("fdtd_mode_apply_beta_squared", m.struct, omega, out.struct)
    b2 = complex(beta.re, beta.im) ** 2
    inner = (slice(2, -2), slice(2, -2), slice(3, 5))
    h, bh = m.fields[inner], out.fields[inner]
    assert b2.real > omega ** 2
    assert np.linalg.norm(bh - b2 * h) <= 1e-4 * np.linalg.norm(b2 * h)
