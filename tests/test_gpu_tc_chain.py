"""Tensor-memory kernels launched back to back, small enough that several of their CTAs fit one SM: each may be set up beside
the one before it, but must not take tensor memory that one still waits for.  The last result is checked against float64; the
TF32 route rounds the operands of two chained products to 10 bits (2e-3 in the repository's tolerance)."""
import numpy as np
import pytest

from gpu_util import TOL, dev, normal, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [32, 64])
@pytest.mark.parametrize("between", [False, True])
def test_dependent_attention_calls(talos, S, between):
    import torch
    ctx, BH, d = talos.torch_context(0), 600, 32
    q, k, v, w = normal(1, (BH, S, d)), normal(2, (BH, S, d)), normal(3, (BH, S, d)), normal(4, (d, d), 0.2)
    tq, tk, tv, tw = dev(q), dev(k), dev(v), dev(w)
    out, mid = torch.empty_like(tq), torch.empty_like(tq)
    P, L = talos.ptr, talos.lib
    for _ in range(50):
        L.talos_attention_fwd(ctx.handle, P(tq), P(tk), P(tv), P(out), None, BH, S, d, d, 0.2, 1, 2)
        if between:
            L.talos_linear_fwd(ctx.handle, P(out), P(tw), None, P(mid), None, BH * S, d, d, 0, 2)
    ctx.synchronize()
    s = np.where(np.tril(np.ones((S, S), bool)), (q @ k.transpose(0, 2, 1)) * 0.2, -np.inf)
    p = np.exp(s - s.max(-1, keepdims=True)); p /= p.sum(-1, keepdims=True)
    assert rel_err(out, p @ v) <= TOL[2]
    if between:
        assert rel_err(mid, p @ v @ w) <= 2 * TOL[2]
