"""Tensor-core products on both sides of the rows at which the tile width changes (148 SMs: 256 columns wide while 128 x 128 tiles would
outnumber the SMs, then 128, then 64), widths that end inside a tile, bias and activation in the epilogue.  Reference float64."""
import ctypes

import numpy as np
import pytest

from gpu_util import TOL, dev, host, normal, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(4736, 256, 128), (4737, 256, 128), (9472, 256, 128), (9473, 252, 96), (3001, 600, 100), (2300, 130, 508), (18945, 128, 64), (512, 1024, 500)])
@pytest.mark.parametrize("opA,opB", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("mode", [1, 2])
def test_product(talos, M, N, K, opA, opB, mode):
    ctx = talos.torch_context(0)
    A, B = normal(1, (K, (M + 3) // 4 * 4) if opA else (M, K)), normal(2, (N, K) if opB else (K, N))
    bias, guard = normal(3, (N,)), 3
    a, b, bi, c = dev(A), dev(B), dev(bias), dev(np.full((M + guard, N), -7.0))
    epi = talos.Epilogue(bias=talos.ptr(bi), act=talos.ACT_TANH)
    talos.lib.talos_gemm(ctx.handle, opA, opB, M, N, K, talos.ptr(a), A.shape[1], talos.ptr(b), B.shape[1], talos.ptr(c), N, mode, ctypes.byref(epi))
    got = host(c)
    ref = (A.T[:M] if opA else A) @ (B.T if opB else B) + bias
    # through tanh only where it is not saturated: the products' standard deviation is sqrt(K)
    plain = dev(np.full((M + guard, N), -7.0))
    talos.lib.talos_gemm(ctx.handle, opA, opB, M, N, K, talos.ptr(a), A.shape[1], talos.ptr(b), B.shape[1], talos.ptr(plain), N, mode, None)
    assert rel_err(host(plain)[:M], ref - bias) <= TOL[mode]
    assert np.abs(got[:M] - np.tanh(ref)).max() <= (1e-4 if mode == 1 else 0.1)
    assert np.all(got[M:] == -7.0) and np.all(host(plain)[M:] == -7.0)


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("M,N,K,opA,slabs", [(65536, 256, 1024, 0, False), (20000, 250, 1032, 0, False), (256, 256, 65536, 1, True), (250, 64, 30000, 1, True)])
def test_split_of_the_reduction(talos, M, N, K, opA, slabs, mode):
    # The reduction is split through memory only where that pays for the slabs' traffic: not for many tiles with a last round
    # that is not full, but for few tiles and a long reduction.  Either way whole chains of the tensor core's sums keep the
    # mode's accuracy.
    import torch
    ctx = talos.torch_context(0)
    g = torch.Generator(device="cuda"); g.manual_seed(5)
    pad = (-M) % 4 if opA else 0
    A = torch.randn((K, M + pad) if opA else (M, K), device="cuda", generator=g); B = torch.randn((K, (N + 3) // 4 * 4), device="cuda", generator=g)
    C = torch.empty(M, N, device="cuda")
    for _ in range(2):                       # a context's first product runs the start-up check's, too
        ctx.timeline_begin()
        talos.lib.talos_gemm(ctx.handle, opA, 0, M, N, K, talos.ptr(A), A.shape[1], talos.ptr(B), B.shape[1], talos.ptr(C), N, mode, None)
    ran = [name for name, _ in ctx.timeline_end()]
    assert ("splitk_reduce" in ran) == slabs and any(name.startswith("gemm_tcgen05") for name in ran), ran
    ref = (A.double().T[:M] if opA else A.double()) @ B[:, :N].double()
    assert float((C.double() - ref).norm() / ref.norm()) <= TOL[mode]
