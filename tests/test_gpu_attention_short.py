"""One-launch attention (attention_short.cu), forward with probabilities and backward from them, where its tiles end: sequences
around 32, 64 and 128, heads around 16, 32 and 64, unequal widths, both masks, every arithmetic mode, few heads and more than
there are SMs, and shapes just outside (odd widths, unaligned heads, more than 64 columns), which take the other routes.  The reference
is float64; fp32 sums of at most 128 + 64 terms behind an exponential stay within a few 1e-6.  The TF32 routes round four operands
of chained products to 10 bits (2^-11 each, 2e-3 for a product in the repository's tolerance); the gradients of Q and K come
out of two of them in a row behind a cancelling difference: twice that."""
import numpy as np
import pytest

from gpu_util import TOL, dev, host, normal, rel_err

pytestmark = pytest.mark.gpu


SHAPES = [(1, 8, 8), (31, 16, 16), (32, 8, 20), (33, 32, 32), (50, 16, 16), (64, 32, 32), (65, 36, 12), (100, 48, 64), (127, 64, 64), (128, 16, 8), (40, 68, 16), (40, 6, 7),
          (17, 4, 4)]


# few heads; unaligned ones; more heads than SMs, on either side of the dispatch
@pytest.mark.parametrize("S,dqk,dv,BH,offset", [s + (5, 0) for s in SHAPES] + [(50, 16, 16, 5, 1)] + [s + (300, 0) for s in SHAPES if s[0] in (64, 65, 100)])
@pytest.mark.parametrize("causal", [0, 1])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_forward_and_backward(talos, S, dqk, dv, BH, offset, causal, mode):
    import torch
    ctx, scale = talos.torch_context(0), 0.3
    q, k, v, do = normal(1, (BH, S, dqk)), normal(2, (BH, S, dqk)), normal(3, (BH, S, dv)), normal(4, (BH, S, dv))
    s = (q @ k.transpose(0, 2, 1)) * scale
    if causal:
        s = np.where(np.tril(np.ones((S, S), bool)), s, -np.inf)
    p = np.exp(s - s.max(-1, keepdims=True)); p /= p.sum(-1, keepdims=True)
    dp = do @ v.transpose(0, 2, 1)
    ds = scale * p * (dp - (dp * p).sum(-1, keepdims=True))
    ref = dict(out=p @ v, probs=p, dq=ds @ k, dk=ds.transpose(0, 2, 1) @ q, dv=p.transpose(0, 2, 1) @ do)
    P = talos.ptr

    def buffer(shape, values=None):     # `offset` floats off a 16-byte boundary, sentinels behind
        n = int(np.prod(shape))
        t = torch.full((offset + n + 4,), 7.0, device="cuda")
        if values is not None:
            t[offset:offset + n] = dev(values).ravel()
        return t, P(t) + 4 * offset

    b = {n: buffer(a.shape, a) for n, a in dict(q=q, k=k, v=v, do=do).items()}
    b.update({n: buffer(a.shape) for n, a in ref.items()})
    t = {n: a for n, (_, a) in b.items()}
    L = talos.lib
    L.talos_attention_fwd(ctx.handle, t["q"], t["k"], t["v"], t["out"], t["probs"], BH, S, dqk, dv, scale, causal, mode)
    L.talos_attention_bwd(ctx.handle, t["q"], t["k"], t["v"], t["probs"], t["do"], t["dq"], t["dk"], t["dv"], BH, S, dqk, dv, scale, mode)
    bare = buffer(ref["out"].shape)
    L.talos_attention_fwd(ctx.handle, t["q"], t["k"], t["v"], bare[1], None, BH, S, dqk, dv, scale, causal, mode)
    ctx.synchronize()
    for n, r in ref.items():
        got = host(b[n][0])[offset:]
        if S == 1 and n in ("dq", "dk"):
            assert np.abs(got[:r.size]).max() <= (1e-5 if mode != 2 else 2e-2)         # exactly zero in real arithmetic
        else:
            tol = TOL[mode] * (2 if mode == 2 and n in ("dq", "dk") else 1)
            assert rel_err(got[:r.size], r.ravel()) <= tol, (n, rel_err(got[:r.size], r.ravel()))
        assert np.all(got[r.size:] == 7.0), n
    assert rel_err(host(bare[0])[offset:offset + ref["out"].size], ref["out"].ravel()) <= TOL[mode]


@pytest.mark.parametrize("mode,dqk,dv,result,source", [(m, 16, 16) + rs for m in (0, 1) for rs in (("out", "q"), ("out", "v"), ("dk", "q"), ("dv", "do"))] +
                         [(1, 32, 16, "out", "q"), (0, 16, 32, "dk", "v"), (1, 16, 32, "dk", "v")])
def test_results_over_inputs(talos, mode, dqk, dv, result, source):
    # Head by head in place: the one-launch kernels.  At another width heads meet each other's: the separate products, whose order
    # allows it (fp32 mode has no such forward: its fused kernel, too, is one CTA a head).
    BH, S, scale = 300, 48, 0.3
    ctx, P, L = talos.torch_context(0), talos.ptr, talos.lib
    a = dict(q=normal(1, (BH, S, dqk)), k=normal(2, (BH, S, dqk)), v=normal(3, (BH, S, dv)), do=normal(4, (BH, S, dv)))
    s = (a["q"] @ a["k"].transpose(0, 2, 1)) * scale
    p = np.exp(s - s.max(-1, keepdims=True)); p /= p.sum(-1, keepdims=True)
    dp = a["do"] @ a["v"].transpose(0, 2, 1)
    ds = scale * p * (dp - (dp * p).sum(-1, keepdims=True))
    ref = dict(out=p @ a["v"], dk=ds.transpose(0, 2, 1) @ a["q"], dv=p.transpose(0, 2, 1) @ a["do"], dq=ds @ a["k"])
    t = {n: dev(x) for n, x in a.items()}
    t.update({n: dev(np.zeros(r.shape)) for n, r in ref.items()}, probs=dev(p))
    t[result] = t[source]
    held, t = t, {n: P(x) for n, x in t.items()}
    if result == "out":
        L.talos_attention_fwd(ctx.handle, t["q"], t["k"], t["v"], t["out"], None, BH, S, dqk, dv, scale, 0, mode)
    else:
        L.talos_attention_bwd(ctx.handle, t["q"], t["k"], t["v"], t["probs"], t["do"], t["dq"], t["dk"], t["dv"], BH, S, dqk, dv, scale, mode)
    ctx.synchronize()
    assert rel_err(host(held[result]).ravel()[:ref[result].size], ref[result].ravel()) <= TOL[mode]
    if result != "out":
        assert rel_err(held["dq"], ref["dq"]) <= TOL[mode]
