"""The small-product kernels (gemm_small.cu) at the sizes where they can go wrong: tile edges (16, 32 and 64 wide), K around
a chunk (128) and around what a cluster splits, widths that rule out 128-bit accesses, every operand layout, and the
one-launch Linear backward with its fused activation derivative and bias gradient.  The reference is float64; fp32 sums of K
terms with round-to-nearest products stay within sqrt(K) * 2^-23 of it in the 2-norm, 1e-5 allows a factor of ten at K = 1 100."""
import ctypes

import numpy as np
import pytest

from gpu_util import TOL, dev, host, normal, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(talos):
    c = talos.torch_context(0)
    yield c
    c.synchronize()


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (15, 17, 5), (16, 16, 128), (33, 31, 129), (64, 64, 64), (65, 4, 300), (40, 36, 1100), (1000, 64, 20),
                                   (2100, 68, 33), (17, 2000, 8), (200, 200, 1025), (9500, 5, 70), (9600, 16, 64), (9700, 65, 33), (9600, 64, 64)])
@pytest.mark.parametrize("opA,opB", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_product(talos, ctx, M, N, K, opA, opB):
    import torch
    A, B = normal(1, (K, M) if opA else (M, K)), normal(2, (N, K) if opB else (K, N))
    bias, C0 = normal(3, (N,)), normal(4, (M, N))
    a, b, bi, c = dev(A), dev(B), dev(bias), dev(np.pad(C0, ((0, 1), (0, 0)), constant_values=-7.0))
    epi = talos.Epilogue(bias=talos.ptr(bi), act=talos.ACT_TANH, beta=1)
    talos.lib.talos_gemm(ctx.handle, opA, opB, M, N, K, talos.ptr(a), A.shape[1], talos.ptr(b), B.shape[1], talos.ptr(c), N, 1, ctypes.byref(epi))
    ref = C0 + np.tanh((A.T if opA else A) @ (B.T if opB else B) + bias)
    got = host(c)
    assert rel_err(got[:M], ref) <= 1e-5
    assert np.all(got[M] == -7.0)                                # nothing past the last row


@pytest.mark.parametrize("M,N,K", [(64, 64, 9001), (64, 64, 65536), (33, 5, 20000), (8, 64, 9000), (16, 16, 40004), (70, 20, 33335), (40, 36, 16384), (300, 12, 16387)])
@pytest.mark.parametrize("opA,opB", [(1, 0), (0, 1)])
def test_long_reduction(talos, ctx, M, N, K, opA, opB):
    # slabs of the reduction whose results go through memory: ends inside a slab and a chunk, every tile of that route, the epilogue
    # behind the sum.  Rounding: sums of K / (slabs * splits * groups) terms, then of those sums; 1e-5 is ten times that.
    import torch
    A, B = normal(1, (K, M) if opA else (M, K)), normal(2, (N, K) if opB else (K, N), 1.0 / np.sqrt(K))
    bias, C0 = normal(3, (N,)), normal(4, (M, N))
    a, b, bi, c = dev(A), dev(B), dev(bias), dev(np.pad(C0, ((0, 1), (0, 0)), constant_values=-7.0))
    epi = talos.Epilogue(bias=talos.ptr(bi), act=talos.ACT_TANH, beta=1)
    args = (ctx.handle, opA, opB, M, N, K, talos.ptr(a), A.shape[1], talos.ptr(b), B.shape[1])
    talos.lib.talos_gemm(*args, talos.ptr(c), N, 0, ctypes.byref(epi))
    ref = (A.T if opA else A) @ (B.T if opB else B)
    got = host(c)
    assert rel_err(got[:M], C0 + np.tanh(ref + bias)) <= 1e-5 and np.all(got[M] == -7.0)
    plain = [torch.empty(M, N, device="cuda:0") for _ in range(2)]
    for p in plain:
        talos.lib.talos_gemm(*args, talos.ptr(p), N, 0, None)
    assert rel_err(plain[0], ref) <= 1e-5 and torch.equal(plain[0], plain[1])


@pytest.mark.parametrize("rows,fin,fout", [(1, 4100, 4096), (16, 2048, 2048), (3, 700, 3000)])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_wide_layer_of_few_rows(talos, ctx, rows, fin, fout, mode):
    # on either side of where a product of few rows is walked too long for these kernels, and dW has more tiles than a round of blocks
    import torch
    x, W, dy = normal(5, (rows, fin)), normal(6, (fin, fout), 0.02), normal(8, (rows, fout))
    tx, tw, ty = dev(x), dev(W), dev(dy)
    y, dx, dW, db = (torch.empty(*s, device="cuda:0") for s in ((rows, fout), (rows, fin), (fin, fout), (fout,)))
    P = talos.ptr
    talos.lib.talos_linear_fwd(ctx.handle, P(tx), P(tw), None, P(y), None, rows, fin, fout, 0, mode)
    talos.lib.talos_linear_bwd(ctx.handle, P(tx), P(tw), None, P(ty), P(dx), P(dW), P(db), rows, fin, fout, 0, mode, 0)
    for got, ref in ((y, x @ W), (dx, dy @ W.T), (dW, x.T @ dy), (db, dy.sum(0))):
        assert rel_err(got, ref) <= TOL[mode]


@pytest.mark.parametrize("rows,fin,fout", [(128, 512, 512), (64, 256, 1024), (2048, 40, 300), (1, 1, 1), (64, 8, 64), (64, 64, 1), (64, 64, 5), (129, 12, 20), (300, 64, 64), (1100, 7, 33), (4096, 8, 16), (500, 256, 256)])
@pytest.mark.parametrize("act", ["none", "tanh", "relu", "silu"])
@pytest.mark.parametrize("parts", ["all", "dx", "dw", "accumulate"])
def test_linear_backward(talos, ctx, rows, fin, fout, act, parts):
    import torch
    x, W, saved, dy = normal(5, (rows, fin)), normal(6, (fin, fout)), np.tanh(normal(7, (rows, fout))), normal(8, (rows, fout))
    saved = saved.astype(np.float32).astype(np.float64)
    if act == "none": d = 1.0
    elif act == "tanh": d = 1 - saved ** 2
    elif act == "relu": d = (saved > 0).astype(np.float64)
    else:
        g = 1 / (1 + np.exp(-saved)); d = g * (1 + saved * (1 - g))
    dz = dy * d
    acc = 7 if parts == "accumulate" else 0
    base = [normal(9, (rows, fin)), normal(10, (fin, fout)), normal(11, (fout,))]
    out = [dev(np.append(b.ravel(), -7.0)) for b in base]
    tx, tw, ts, ty = dev(x), dev(W), dev(saved), dev(dy)
    want = [parts != "dw", parts != "dx", parts != "dx"]
    talos.lib.talos_linear_bwd(ctx.handle, talos.ptr(tx), talos.ptr(tw), talos.ptr(ts), talos.ptr(ty), *[talos.ptr(o) if w else None for o, w in zip(out, want)],
                               rows, fin, fout, talos.ACTS[act], 1, acc)
    ref = [dz @ W.T, x.T @ dz, dz.sum(0)]
    for o, r, b, w in zip(out, ref, base, want):
        got = host(o)
        assert got[-1] == -7.0
        if w:
            # the column sum of N(0, 1)-sized terms can be far smaller than its terms: their own size is part of the bound
            r = r + b if acc else r
            err = np.linalg.norm(got[:-1].reshape(r.shape) - r)
            assert err <= 1e-5 * max(np.linalg.norm(r), np.sqrt(r.size)), (err, np.linalg.norm(r))
        else:
            assert np.array_equal(got[:-1], b.ravel().astype(np.float32))


@pytest.mark.parametrize("rows,act", [(64, "tanh"), (64, "none"), (5000, "silu")])
@pytest.mark.parametrize("mode", [0, 1])
def test_linear_backward_of_nothing(talos, ctx, rows, act, mode):
    # every result may be left out, also all of them
    x, W, dy = dev(normal(5, (rows, 16))), dev(normal(6, (16, 24))), dev(normal(7, (rows, 24)))
    talos.lib.talos_linear_bwd(ctx.handle, talos.ptr(x), talos.ptr(W), talos.ptr(dy), talos.ptr(dy), None, None, None, rows, 16, 24, talos.ACTS[act], mode, 0)
    ctx.synchronize()


@pytest.mark.parametrize("over", ["dW over W", "dW over dy", "dW over saved", "db over dy", "db over saved"])
@pytest.mark.parametrize("mode", [0, 1])
def test_linear_backward_over_its_inputs(talos, ctx, over, mode):
    # results over inputs that the steps before them have already used (dZ is a copy here, dX comes before dW and db)
    n = 200
    x, W, saved, dy = normal(5, (n, n)), normal(6, (n, n)), np.tanh(normal(7, (n, n))), normal(8, (n, n))
    saved = saved.astype(np.float32).astype(np.float64)
    dz = dy * (1 - saved ** 2)
    t = dict(x=dev(x), W=dev(W), saved=dev(saved), dy=dev(dy))
    out = dict(dx=dev(np.zeros((n, n))), dW=dev(np.zeros((n, n))), db=dev(np.zeros(n)))
    result, source = over.split(" over ")
    out[result] = t[source]
    p = {k: talos.ptr(v) for k, v in {**t, **out}.items()}
    talos.lib.talos_linear_bwd(ctx.handle, talos.ptr(t["x"]), talos.ptr(t["W"]), talos.ptr(t["saved"]), talos.ptr(t["dy"]), p["dx"], p["dW"], p["db"], n, n, n,
                               talos.ACTS["tanh"], mode, 0)
    assert rel_err(out["dx"], dz @ W.T) <= 1e-5 and rel_err(out["dW"], x.T @ dz) <= 1e-5
    assert np.abs(host(out["db"]).ravel()[:n] - dz.sum(0)).max() <= 1e-5 * np.sqrt(n) * 4


@pytest.mark.parametrize("rows,width,modes", [(1, 8, (0, 1, 2)), (70, 36, (0, 1, 2)), (300, 64, (0, 1, 2)), (20000, 64, (0, 1, 2)), (33, 5, (0, 1, 2)),
                                              (500, 128, (0, 1, 2)), (4736, 256, (1, 2)), (9000, 252, (1, 2))])
@pytest.mark.parametrize("what", ["y", "z_save"])
def test_square_linear_in_place(talos, ctx, rows, width, modes, what):
    # y (or z_save) over x: one tile has to span the columns (64 on the CUDA cores, 128 for many rows, 256 on the tensor cores)
    import torch
    x, W, b = normal(5, (rows, width)), normal(6, (width, width), 1.0 / np.sqrt(width)), normal(7, (width,), 0.1)
    w, bias, other = dev(W), dev(b), torch.empty(rows, width, device="cuda:0")
    z = x @ W + b
    for mode in modes:
        io = dev(x)
        y, save = (io, other) if what == "y" else (other, io)
        talos.lib.talos_linear_fwd(ctx.handle, talos.ptr(io), talos.ptr(w), talos.ptr(bias), talos.ptr(y), talos.ptr(save), rows, width, width, talos.ACTS["tanh"], mode)
        assert rel_err(save, z) <= TOL[mode] and rel_err(y, np.tanh(z)) <= TOL[mode], mode


@pytest.mark.needs_tensor_cores
@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("M,N,K", [(200, 72, 40), (129, 33, 100), (1000, 36, 520), (64, 260, 64)])
def test_both_routes_of_a_small_product(talos, ctx, M, N, K, mode, monkeypatch):
    # the tensor-core kernels stay in use for products of this size that bring prepared weights (the PPO trainer's)
    import torch
    A, B = normal(12, (M, K)), normal(13, (K, (N + 3) // 4 * 4))
    a, b, c = dev(A), dev(B), torch.empty(M, N, device="cuda:0")
    for route, tol in (("small", 1e-5), ("tensor", 1e-5 if mode == 1 else 2e-3)):
        if route == "tensor":
            monkeypatch.setenv("TALOS_TC_NO_SMALL", "1")
        talos.lib.talos_gemm(ctx.handle, 0, 0, M, N, K, talos.ptr(a), K, talos.ptr(b), B.shape[1], talos.ptr(c), N, mode, None)
        assert rel_err(c, A @ B[:, :N]) <= tol, route
