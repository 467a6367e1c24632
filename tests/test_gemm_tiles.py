"""The tcgen05 GEMM's tile edges (umma_gemm.cu) and the network's grouped
launches at batches that leave ragged tiles.

Products: |C - C_ref| <= (K + 8) 2^-22 |A| |B|^T element by element (K FP32
additions of exact BF16 products, each rounded to 2^-24 relative at worst
twice, with a factor of two to spare).  Gradients: against the restatement with
the same BF16 rounding points, within the bounds its own test uses."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import surrogate as S

torch = pytest.importorskip("torch")
FP = C.POINTER(C.c_float)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (127, 31, 16), (129, 33, 72), (128, 32, 256), (130, 40, 264),
                                   (4100, 300, 328), (8192, 640, 64)])
def test_gemm_tile_edges(fd, gpu, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    B = torch.randn(N, K, generator=g).to(torch.bfloat16).cuda()
    out = torch.full((M, N), 7.0, dtype=torch.float32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    fd.call("fdtd_gemm_bf16", A.data_ptr(), K, B.data_ptr(), K, M, N, K, None, 0, 1.0, 0.0, out.data_ptr(), N, None, N,
            None, N, err.data_ptr(), None)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = A.double() @ B.double().T
    bound = (K + 8) * 2.0 ** -22 * (A.double().abs() @ B.double().abs().T)
    assert bool(((out.double() - ref).abs() <= bound).all())


@pytest.mark.gpu
@pytest.mark.parametrize("B,hid,nin,nout", [(8, 8, 3, 2), (136, 40, 20, 22), (392, 264, 9, 33)])
def test_network_gradients_at_ragged_sizes(fd, gpu, B, hid, nin, nout):
    net = fd.lib.fdtd_mlp_new(nin, hid, nout, 5)
    assert net
    rng = np.random.default_rng(B)
    x, t = (rng.normal(size=(B, n)).astype(np.float32) for n in (nin, nout))
    flat = np.zeros(fd.lib.fdtd_mlp_param_count(net), np.float32)
    fd.call("fdtd_mlp_get_params", net, flat.ctypes.data_as(FP))
    grad, dx, loss = np.zeros_like(flat), np.zeros_like(x), C.c_double()
    fd.call("fdtd_mlp_gradients", net, x.ctypes.data_as(FP), t.ctypes.data_as(FP), B, grad.ctypes.data_as(FP),
            C.byref(loss))
    fd.call("fdtd_mlp_input_gradient", net, x.ctypes.data_as(FP), t.ctypes.data_as(FP), B, dx.ctypes.data_as(FP))
    fd.lib.fdtd_mlp_free(net)
    P = S.unflatten(flat.astype(np.float64), nin, hid, nout)
    ref_loss, ref, _ = S.gradients(P, x.astype(np.float64), t.astype(np.float64))
    assert abs(loss.value - ref_loss) < 1e-3 * ref_loss
    for got, want in zip(S.unflatten(grad.astype(np.float64), nin, hid, nout), ref):
        for a, b in zip(got, want):
            assert np.abs(a - b).max() < 2e-2 * np.abs(b).max()
    want = S.input_gradient(P, x.astype(np.float64), t.astype(np.float64))
    assert np.abs(dx - want).max() < 2e-2 * np.abs(want).max()
