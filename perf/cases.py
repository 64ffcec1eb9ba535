"""Performance cases of the framework: what its users have it do, through its public entry points.

Eight kinds of work over the sizes of the repository's own benchmark configurations, tests and shipped settings (8
observations, hidden 64, 5 actions, 2 048 steps an update in minibatches of 256) up to its largest one (1 048 576
transitions in minibatches of 65 536), in the three arithmetic modes a caller can choose:

  update    the learning phase of PPO: log-probabilities of the stored actions, then the epochs x minibatches loops
  rollout   one policy step of the latent-attention actor for many simulations at once, each with its own KV ring
  block     transformer block forward + backward (RMSNorm, QKV, RoPE, causal attention, SiLU MLP, residuals)
  mla       latent-attention layer forward over whole sequences (inference)
  mlp       Linear layers forward + backward with biases and an activation
  matmul    a matrix product and its two backward products
  gae       advantage estimation over a rollout buffer: reverse scan, then normalisation
  dqn       one dueling double-DQN train step
"""
import importlib
import math

import numpy as np
import torch

talos = importlib.import_module("talos-xii_b200")
L, P = talos.lib, talos.ptr
MODES = talos.MODES
_CTX = {}


def _ctx():
    """The one context a program creates at start-up, on torch's current stream."""
    if "ctx" not in _CTX:
        _CTX["ctx"] = talos.torch_context(0)
    return _CTX["ctx"]


def listed():
    return [
        # the shipped PPO settings: a 2 048-step rollout, 8 epochs of minibatch 256, 8 observations, 5 actions -- 64 tiny dependent steps
        dict(name="update_shipped", kind="update", n=2048, minibatch=256, epochs=8, obs=8, hidden=64, actions=5, mode="tf32x3", host=False),
        # a mid-sized rollout that does not divide into its minibatches, in the fast mode, transitions already on the GPU
        dict(name="update_ragged", kind="update", n=50001, minibatch=8192, epochs=3, obs=64, hidden=256, actions=16, mode="tf32", host=False),
        # the benchmark's update, end to end: 1 048 576 transitions from pinned host buffers, 4 epochs of minibatch 65 536
        dict(name="update_large", kind="update", n=1048576, minibatch=65536, epochs=4, obs=64, hidden=256, actions=16, mode="tf32x3", host=True),
        # one pull of a small batch of simulations: twenty dependent small calls, latency is all there is
        dict(name="rollout_small", kind="rollout", sims=64, hidden=64, context=16, mode="tf32x3"),
        # one pull of a whole population of simulations
        dict(name="rollout_large", kind="rollout", sims=65536, hidden=64, context=16, mode="tf32x3"),
        # training step of the benchmark's transformer block: batch 1 024 x 64 tokens, width 256, 8 heads
        dict(name="block_train", kind="block", batch=1024, seq=64, width=256, heads=8, mode="tf32x3"),
        # the same block on a small batch whose sequence length fits no tile
        dict(name="block_ragged", kind="block", batch=24, seq=50, width=64, heads=4, mode="tf32"),
        # inference of the benchmark's latent-attention layer: batch 512 x 128 tokens, width 512, rank 64, 8 heads of 64 + 32
        dict(name="mla_forward", kind="mla", batch=512, seq=128, width=512, rank=64, heads=8, head=64, rope=32, mode="tf32"),
        # the benchmark's MLP, forward and backward: 8 192 observations through 64-256-256-16
        dict(name="mlp_train", kind="mlp", rows=8192, obs=64, hidden=256, out=16, act="tanh", mode="tf32x3"),
        # the benchmark's large product and both its backward products
        dict(name="matmul_large", kind="matmul", m=4096, n=4096, k=4096, mode="tf32"),
        # advantages of a 1 048 576-step rollout buffer
        dict(name="gae_buffer", kind="gae", n=1048576),
        # the DQN agent's train step at its replay batch of 64: two dozen tiny dependent calls
        dict(name="dqn_step", kind="dqn", batch=64, obs=8, hidden=64, actions=5, mode="tf32x3"),
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]; about half of them odd."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v))


def draw(rng):
    kind = rng.choice(["update", "update", "update", "rollout", "rollout", "block", "block", "mla", "mlp", "matmul", "gae", "dqn"])
    mode = rng.choice(["tf32x3", "tf32x3", "tf32x3", "tf32", "tf32", "fp32"])
    if kind == "update":
        if rng.random() < 0.5:      # policies of the shipped size
            n = _log(rng, 512, 8192)
            return dict(kind=kind, n=n, minibatch=min(n, _log(rng, 64, 1024)), epochs=rng.randint(2, 10), obs=rng.choice([8, 8, 12, 16]), hidden=64,
                        actions=rng.choice([5, 5, 4, 8]), mode=mode, host=rng.random() < 0.3)
        n = _log(rng, 16384, 65536 if mode == "fp32" else 524288)
        return dict(kind=kind, n=n, minibatch=min(n, _log(rng, 2048, 65536)), epochs=rng.randint(1, 4), obs=rng.choice([32, 64, 64]),
                    hidden=rng.choice([128, 256, 256]), actions=rng.choice([5, 16, 16]), mode=mode, host=rng.random() < 0.3)
    if kind == "rollout":
        return dict(kind=kind, sims=_log(rng, 1, 65536), hidden=rng.choice([64, 64, 128]), context=rng.randint(4, 16), mode=mode)
    if kind == "block":
        seq = rng.randint(8, 128)
        seq = rng.choice([seq, (seq + 31) // 32 * 32])
        width, heads = rng.choice([(64, 4), (128, 4), (256, 8)])
        return dict(kind=kind, batch=_log(rng, 4, max(4, (16384 if mode == "fp32" else 65536) // seq)), seq=seq, width=width, heads=heads, mode=mode)
    if kind == "mla":
        seq = rng.randint(16, 128)
        seq = rng.choice([seq, (seq + 31) // 32 * 32])
        width, rank, heads, head, rope = rng.choice([(64, 32, 4, 16, 16), (256, 64, 8, 32, 32), (512, 64, 8, 64, 32)])
        return dict(kind=kind, batch=_log(rng, 4, 512), seq=seq, width=width, rank=rank, heads=heads, head=head, rope=rope, mode=mode)
    if kind == "mlp":
        return dict(kind=kind, rows=_log(rng, 64, 65536), obs=rng.choice([8, 64]), hidden=rng.choice([64, 256]), out=rng.choice([5, 16]),
                    act=rng.choice(["tanh", "relu", "silu"]), mode=mode)
    if kind == "matmul":
        top = 2048 if mode == "fp32" else 4096
        sizes = [_log(rng, 128, top) for _ in range(3)]
        if rng.random() < 0.7:
            sizes = [(s + 3) // 4 * 4 for s in sizes]
        return dict(kind=kind, m=sizes[0], n=sizes[1], k=sizes[2], mode=mode)
    if kind == "gae":
        return dict(kind=kind, n=_log(rng, 2048, 4194304))
    return dict(kind=kind, batch=_log(rng, 32, 2048), obs=rng.choice([8, 16]), hidden=rng.choice([64, 128]), actions=rng.choice([5, 8]), mode=mode)


# ---- states: inputs, weights, result buffers and handles a program keeps between calls ----------------------------------


class _State:
    pass


class _Inputs:
    """Seeded values on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def normal(self, *shape, std=1.0):
        return torch.randn(*shape, device="cuda", generator=self.g) * std

    def uniform(self, *shape, lim=1.0):
        return (torch.rand(*shape, device="cuda", generator=self.g) * 2 - 1) * lim

    def xavier(self, fi, fo):
        return self.uniform(fi, fo, lim=math.sqrt(6.0 / (fi + fo)))

    def ints(self, n, high):
        return torch.randint(0, high, (n,), device="cuda", generator=self.g, dtype=torch.int32)

    def chance(self, n, p):
        return (torch.rand(n, device="cuda", generator=self.g) < p).to(torch.int32)


def _empty(*shape):
    return torch.empty(*shape, device="cuda")


class _Trainer(_State):
    def __del__(self):
        self.trainer.close()


def _prepare_update(c, seed):
    s, r, ctx = _Trainer(), _Inputs(seed), _ctx()
    n, o, h, a = c["n"], c["obs"], c["hidden"], c["actions"]
    s.n, s.epochs, s.host = n, c["epochs"], c["host"]
    s.trainer = talos.PPOTrainer(ctx, talos.PpoConfig(o, h, a, c["minibatch"], MODES[c["mode"]]))
    weights = [r.xavier(o, h), torch.zeros(h), r.xavier(h, h), torch.zeros(h), r.xavier(h, a), torch.zeros(a), r.xavier(h, 1), torch.zeros(1)]
    s.trainer.set_params(np.concatenate([w.cpu().numpy().ravel() for w in weights]))
    s.obs, s.actions, s.adv, s.ret, s.old = r.normal(n, o), r.ints(n, a), r.normal(n), r.normal(n), _empty(n)
    if s.host:      # the rollout workers stored the log-probabilities with the transitions, in pinned memory
        s.trainer.log_prob(s.obs, s.actions, n, s.old)
        ctx.synchronize()
        s.obs, s.actions, s.adv, s.ret, s.old = (t.cpu().pin_memory() for t in (s.obs, s.actions, s.adv, s.ret, s.old))
    s.params = np.empty(s.trainer.n_params, dtype=np.float32)
    return s


def _run_update(s):
    if not s.host:
        s.trainer.log_prob(s.obs, s.actions, s.n, s.old)
    s.trainer.update(s.obs, s.actions, s.old, s.adv, s.ret, s.n, s.epochs, host=s.host)
    L.talos_ppo_get_params_host(s.trainer.handle, P(s.params))      # the new weights, as the program hands them to its simulators
    return s.params


def _prepare_rollout(c, seed):
    s, r, ctx = _State(), _Inputs(seed), _ctx()
    n, d, cap = c["sims"], c["hidden"], c["context"] + 1
    heads, rank, dr, obs, acts = 4, 32, 16, 8, 5
    dh = d // heads
    s.n, s.d, s.cap, s.heads, s.rank, s.dr, s.dh, s.obs, s.acts, s.mode = n, d, cap, heads, rank, dr, dh, obs, acts, MODES[c["mode"]]
    s.ctx, s.step, s.scale = ctx.handle, 0, 1.0 / math.sqrt(dh + dr)
    dims = dict(embed=(obs, d), w_dkv=(d, rank), w_uk=(rank, d), w_uv=(rank, d), w_kr=(d, heads * dr), w_q=(d, d), w_qr=(d, heads * dr), w_o=(d, d),
                ffn_1=(d, 2 * d), ffn_2=(2 * d, d), out_proj=(d, d), actor=(d, acts))
    s.dims, s.w = dims, {k: r.xavier(*v) for k, v in dims.items()}
    s.b = {k: r.uniform(dims[k][1], lim=0.05) for k in ("embed", "ffn_1", "ffn_2", "out_proj", "actor")}
    s.gamma = torch.ones(d, device="cuda")
    s.cos, s.sin = _empty(256 * dr // 2), _empty(256 * dr // 2)
    L.talos_rope_table(ctx.handle, dr, 256, 10000.0, P(s.cos), P(s.sin))
    s.states = r.normal(n, obs, std=0.5)
    s.pos = r.ints(n, 90)                                # simulations at different pulls of their episodes
    s.resets = [r.chance(n, 1.0 / 60.0) for _ in range(8)]      # episodes that end with this pull
    s.k_cache, s.v_cache = r.normal(n, heads, cap, dh + dr, std=0.5), r.normal(n, heads, cap, dh, std=0.5)
    s.buf = {k: _empty(n, w) for k, w in dict(h=d, hn=d, c_kv=rank, k_c=d, v_c=d, k_r=heads * dr, q_c=d, q_r=heads * dr, att=d, ao=d, h2=d, f1=2 * d, f2=d, h3=d,
                                              o=d, logits=acts, probs=acts).items()}
    s.p = {k: P(t) for k, t in s.buf.items()}
    s.wp, s.bp = {k: P(t) for k, t in s.w.items()}, {k: P(s.b[k]) if k in s.b else None for k in dims}
    return s


def _run_rollout(s):
    c, n, d, p, mode = s.ctx, s.n, s.d, s.p, s.mode
    gamma = P(s.gamma)

    def linear(name, x, y, act=talos.ACT_NONE):
        L.talos_linear_fwd(c, x, s.wp[name], s.bp[name], y, None, n, s.dims[name][0], s.dims[name][1], act, mode)

    linear("embed", P(s.states), p["h"])
    L.talos_rmsnorm_fwd(c, p["h"], gamma, 1e-5, n, d, p["hn"], None)
    linear("w_dkv", p["hn"], p["c_kv"])
    linear("w_uk", p["c_kv"], p["k_c"])
    linear("w_uv", p["c_kv"], p["v_c"])
    linear("w_kr", p["hn"], p["k_r"])
    linear("w_q", p["hn"], p["q_c"])
    linear("w_qr", p["hn"], p["q_r"])
    L.talos_mla_decode_step(c, p["q_c"], p["q_r"], p["k_c"], p["k_r"], p["v_c"], P(s.cos), P(s.sin), 256 * s.dr // 2, P(s.pos), P(s.k_cache), P(s.v_cache),
                            p["att"], n, s.heads, s.dh, s.dr, s.cap, s.scale)
    linear("w_o", p["att"], p["ao"])
    L.talos_eltwise_binary(c, talos.EW["add"], p["h"], p["ao"], p["h2"], n * d)
    L.talos_rmsnorm_fwd(c, p["h2"], gamma, 1e-5, n, d, p["hn"], None)
    linear("ffn_1", p["hn"], p["f1"], talos.ACT_RELU)
    linear("ffn_2", p["f1"], p["f2"])
    L.talos_eltwise_binary(c, talos.EW["add"], p["h2"], p["f2"], p["h3"], n * d)
    L.talos_rmsnorm_fwd(c, p["h3"], gamma, 1e-5, n, d, p["hn"], None)
    linear("out_proj", p["hn"], p["o"])
    linear("actor", p["o"], p["logits"])
    L.talos_softmax_fwd(c, p["logits"], p["probs"], n, s.acts, 1.0, 0)
    L.talos_decode_advance(c, P(s.pos), P(s.resets[s.step % len(s.resets)]), n)
    s.step += 1
    return {"probs": s.buf["probs"], "pos": s.pos, "k_cache": s.k_cache, "v_cache": s.v_cache}


def _shape4(*v):
    return np.array(v, dtype=np.int64)


def _prepare_block(c, seed):
    s, r, ctx = _State(), _Inputs(seed), _ctx()
    b, q, d, h = c["batch"], c["seq"], c["width"], c["heads"]
    t, f, dh = b * q, 4 * d, d // h
    s.b, s.q, s.d, s.h, s.t, s.f, s.dh, s.mode, s.ctx = b, q, d, h, t, f, dh, MODES[c["mode"]], ctx.handle
    s.x, s.dy = r.normal(t, d), r.normal(t, d)
    s.g1, s.g2 = 1 + r.normal(d, std=0.05), 1 + r.normal(d, std=0.05)
    s.w = {k: r.normal(*v, std=0.02) for k, v in dict(qkv=(d, 3 * d), o=(d, d), f1=(d, f), f2=(f, d)).items()}
    s.cos, s.sin = _empty(q * dh // 2), _empty(q * dh // 2)
    L.talos_rope_table(ctx.handle, dh, q, 10000.0, P(s.cos), P(s.sin))
    wide = dict(n1=d, qkv=3 * d, q=d, kv=2 * d, k=d, v=d, qr=d, kr=d, qh=d, kh=d, vh=d, oh=d, att=d, ao=d, h2=d, n2=d, z=f, f=f, fo=d, y=d,
                df=f, dn2=d, dh2=d, datt=d, doh=d, dqh=d, dkh=d, dvh=d, dqr=d, dkr=d, dv=d, dq=d, dk=d, dkv=2 * d, dqkv=3 * d, dn1=d, dx=d)
    s.buf = {k: _empty(t, w) for k, w in wide.items()}
    s.buf["probs"], s.buf["inv1"], s.buf["inv2"] = _empty(b * h, q, q), _empty(t), _empty(t)
    for k, w in s.w.items():
        s.buf["dw_" + k] = torch.empty_like(w)
    s.buf["dg1"], s.buf["dg2"] = _empty(d), _empty(d)
    s.p = {k: P(v) for k, v in s.buf.items()}
    s.bshd, s.bhsd = _shape4(b, q, h, dh), _shape4(b, h, q, dh)
    return s


def _run_block(s):
    c, t, d, f, m, p, w = s.ctx, s.t, s.d, s.f, s.mode, s.p, s.w
    b, q, h, dh = s.b, s.q, s.h, s.dh
    x, dy, cos, sin, table = P(s.x), P(s.dy), P(s.cos), P(s.sin), q * dh // 2
    none, silu, add, scale = talos.ACT_NONE, talos.ACT_SILU, talos.EW["add"], 1.0 / math.sqrt(dh)
    bshd, bhsd = P(s.bshd), P(s.bhsd)
    # forward
    L.talos_rmsnorm_fwd(c, x, P(s.g1), 1e-6, t, d, p["n1"], p["inv1"])
    L.talos_linear_fwd(c, p["n1"], P(w["qkv"]), None, p["qkv"], None, t, d, 3 * d, none, m)
    L.talos_split_last(c, p["qkv"], p["q"], p["kv"], t, d, 2 * d, 0)
    L.talos_split_last(c, p["kv"], p["k"], p["v"], t, d, d, 0)
    L.talos_rope(c, p["q"], p["qr"], cos, sin, table, b, q, h, dh, 0, 0, 0)
    L.talos_rope(c, p["k"], p["kr"], cos, sin, table, b, q, h, dh, 0, 0, 0)
    L.talos_transpose(c, p["qr"], p["qh"], bshd, 4, 1, 2, 0)
    L.talos_transpose(c, p["kr"], p["kh"], bshd, 4, 1, 2, 0)
    L.talos_transpose(c, p["v"], p["vh"], bshd, 4, 1, 2, 0)
    L.talos_attention_fwd(c, p["qh"], p["kh"], p["vh"], p["oh"], p["probs"], b * h, q, dh, dh, scale, 1, m)
    L.talos_transpose(c, p["oh"], p["att"], bhsd, 4, 1, 2, 0)
    L.talos_linear_fwd(c, p["att"], P(w["o"]), None, p["ao"], None, t, d, d, none, m)
    L.talos_eltwise_binary(c, add, x, p["ao"], p["h2"], t * d)
    L.talos_rmsnorm_fwd(c, p["h2"], P(s.g2), 1e-6, t, d, p["n2"], p["inv2"])
    L.talos_linear_fwd(c, p["n2"], P(w["f1"]), None, p["f"], p["z"], t, d, f, silu, m)
    L.talos_linear_fwd(c, p["f"], P(w["f2"]), None, p["fo"], None, t, f, d, none, m)
    L.talos_eltwise_binary(c, add, p["h2"], p["fo"], p["y"], t * d)
    # backward
    L.talos_linear_bwd(c, p["f"], P(w["f2"]), None, dy, p["df"], p["dw_f2"], None, t, f, d, none, m, 0)
    L.talos_linear_bwd(c, p["n2"], P(w["f1"]), p["z"], p["df"], p["dn2"], p["dw_f1"], None, t, d, f, silu, m, 0)
    L.talos_copy_device(c, p["dh2"], dy, 4 * t * d)
    L.talos_rmsnorm_bwd(c, p["dn2"], p["h2"], P(s.g2), p["inv2"], t, d, p["dh2"], p["dg2"], 1)
    L.talos_linear_bwd(c, p["att"], P(w["o"]), None, p["dh2"], p["datt"], p["dw_o"], None, t, d, d, none, m, 0)
    L.talos_transpose(c, p["datt"], p["doh"], bshd, 4, 1, 2, 0)
    L.talos_attention_bwd(c, p["qh"], p["kh"], p["vh"], p["probs"], p["doh"], p["dqh"], p["dkh"], p["dvh"], b * h, q, dh, dh, scale, m)
    L.talos_transpose(c, p["dqh"], p["dqr"], bhsd, 4, 1, 2, 0)
    L.talos_transpose(c, p["dkh"], p["dkr"], bhsd, 4, 1, 2, 0)
    L.talos_transpose(c, p["dvh"], p["dv"], bhsd, 4, 1, 2, 0)
    L.talos_rope(c, p["dqr"], p["dq"], cos, sin, table, b, q, h, dh, 0, 1, 0)
    L.talos_rope(c, p["dkr"], p["dk"], cos, sin, table, b, q, h, dh, 0, 1, 0)
    L.talos_concat_last(c, p["dk"], p["dv"], p["dkv"], t, d, d)
    L.talos_concat_last(c, p["dq"], p["dkv"], p["dqkv"], t, d, 2 * d)
    L.talos_linear_bwd(c, p["n1"], P(w["qkv"]), None, p["dqkv"], p["dn1"], p["dw_qkv"], None, t, d, 3 * d, none, m, 0)
    L.talos_copy_device(c, p["dx"], p["dh2"], 4 * t * d)
    L.talos_rmsnorm_bwd(c, p["dn1"], x, P(s.g1), p["inv1"], t, d, p["dx"], p["dg1"], 1)
    return {k: s.buf[k] for k in ("y", "dx", "dg1", "dg2", "dw_qkv", "dw_o", "dw_f1", "dw_f2")}


def _prepare_mla(c, seed):
    s, r, ctx = _State(), _Inputs(seed), _ctx()
    b, q, d, rank, h, dh, dr = c["batch"], c["seq"], c["width"], c["rank"], c["heads"], c["head"], c["rope"]
    t = b * q
    s.b, s.q, s.d, s.rank, s.h, s.dh, s.dr, s.t, s.mode, s.ctx = b, q, d, rank, h, dh, dr, t, MODES[c["mode"]], ctx.handle
    s.dims = dict(dkv=(d, rank), uk=(rank, h * dh), uv=(rank, h * dh), q=(d, h * dh), kr=(d, h * dr), qr=(d, h * dr), o=(h * dh, d))
    s.x, s.w = r.normal(t, d), {k: r.normal(*v, std=0.02) for k, v in s.dims.items()}
    s.cos, s.sin = _empty(q * dr // 2), _empty(q * dr // 2)
    L.talos_rope_table(ctx.handle, dr, q, 10000.0, P(s.cos), P(s.sin))
    wide = dict(ckv=rank, kc=h * dh, vc=h * dh, kr=h * dr, qc=h * dh, qr=h * dr, krot=h * dr, qrot=h * dr, qcat=h * (dh + dr), kcat=h * (dh + dr),
                qh=h * (dh + dr), kh=h * (dh + dr), vh=h * dh, oh=h * dh, att=h * dh, y=d)
    s.buf = {k: _empty(t, w) for k, w in wide.items()}
    s.p, s.wp = {k: P(v) for k, v in s.buf.items()}, {k: P(v) for k, v in s.w.items()}
    s.qk_shape, s.v_shape, s.o_shape = _shape4(b, q, h, dh + dr), _shape4(b, q, h, dh), _shape4(b, h, q, dh)
    return s


def _run_mla(s):
    c, t, b, q, h, dh, dr, p, mode = s.ctx, s.t, s.b, s.q, s.h, s.dh, s.dr, s.p, s.mode
    x, cos, sin, table = P(s.x), P(s.cos), P(s.sin), q * dr // 2

    def linear(name, x, y):
        L.talos_linear_fwd(c, x, s.wp[name], None, y, None, t, s.dims[name][0], s.dims[name][1], talos.ACT_NONE, mode)

    linear("dkv", x, p["ckv"])
    linear("uk", p["ckv"], p["kc"])
    linear("uv", p["ckv"], p["vc"])
    linear("kr", x, p["kr"])
    linear("q", x, p["qc"])
    linear("qr", x, p["qr"])
    L.talos_rope(c, p["kr"], p["krot"], cos, sin, table, b, q, h, dr, 0, 0, 0)
    L.talos_rope(c, p["qr"], p["qrot"], cos, sin, table, b, q, h, dr, 0, 0, 0)
    L.talos_concat_last(c, p["qc"], p["qrot"], p["qcat"], t * h, dh, dr)
    L.talos_concat_last(c, p["kc"], p["krot"], p["kcat"], t * h, dh, dr)
    L.talos_transpose(c, p["qcat"], p["qh"], P(s.qk_shape), 4, 1, 2, 0)
    L.talos_transpose(c, p["kcat"], p["kh"], P(s.qk_shape), 4, 1, 2, 0)
    L.talos_transpose(c, p["vc"], p["vh"], P(s.v_shape), 4, 1, 2, 0)
    L.talos_attention_fwd(c, p["qh"], p["kh"], p["vh"], p["oh"], None, b * h, q, dh + dr, dh, 1.0 / math.sqrt(dh + dr), 0, mode)
    L.talos_transpose(c, p["oh"], p["att"], P(s.o_shape), 4, 1, 2, 0)
    linear("o", p["att"], p["y"])
    return s.buf["y"]


def _prepare_mlp(c, seed):
    s, r, ctx = _State(), _Inputs(seed), _ctx()
    s.rows, s.mode, s.ctx, s.act = c["rows"], MODES[c["mode"]], ctx.handle, talos.ACTS[c["act"]]
    dims = [c["obs"], c["hidden"], c["hidden"], c["out"]]
    s.layers = []
    s.x, s.dy = r.normal(s.rows, dims[0]), r.normal(s.rows, dims[-1])
    for i in range(3):
        e = _State()
        fi, fo = dims[i], dims[i + 1]
        e.fi, e.fo, e.act = fi, fo, s.act if i < 2 else talos.ACT_NONE
        e.w, e.b, e.y, e.dx, e.dw, e.db = r.xavier(fi, fo), r.uniform(fo, lim=0.05), _empty(s.rows, fo), _empty(s.rows, fi), _empty(fi, fo), _empty(fo)
        e.z = _empty(s.rows, fo) if e.act == talos.ACT_SILU else None
        s.layers.append(e)
    return s


def _run_mlp(s):
    x = s.x
    for e in s.layers:
        L.talos_linear_fwd(s.ctx, P(x), P(e.w), P(e.b), P(e.y), P(e.z), s.rows, e.fi, e.fo, e.act, s.mode)
        x = e.y
    dy = s.dy
    for i in (2, 1, 0):
        e = s.layers[i]
        x = s.layers[i - 1].y if i else s.x
        L.talos_linear_bwd(s.ctx, P(x), P(e.w), P(e.y if e.z is None else e.z), P(dy), P(e.dx), P(e.dw), P(e.db), s.rows, e.fi, e.fo, e.act, s.mode, 0)
        dy = e.dx
    return [s.layers[2].y, s.layers[0].dx] + [e.dw for e in s.layers] + [e.db for e in s.layers]


def _prepare_matmul(c, seed):
    s, r, ctx = _State(), _Inputs(seed), _ctx()
    m, n, k = c["m"], c["n"], c["k"]
    s.m, s.n, s.k, s.mode, s.ctx = m, n, k, MODES[c["mode"]], ctx.handle
    s.a, s.b, s.g = r.uniform(m, k), r.uniform(k, n), r.uniform(m, n)
    s.c, s.da, s.db = _empty(m, n), _empty(m, k), _empty(k, n)
    return s


def _run_matmul(s):
    m, n, k = s.m, s.n, s.k
    L.talos_gemm(s.ctx, 0, 0, m, n, k, P(s.a), k, P(s.b), n, P(s.c), n, s.mode, None)
    L.talos_gemm(s.ctx, 0, 1, m, k, n, P(s.g), n, P(s.b), n, P(s.da), k, s.mode, None)
    L.talos_gemm(s.ctx, 1, 0, k, n, m, P(s.a), k, P(s.g), n, P(s.db), n, s.mode, None)
    return s.c, s.da, s.db


def _prepare_gae(c, seed):
    s, r, ctx = _State(), _Inputs(seed), _ctx()
    n = c["n"]
    s.n, s.ctx = n, ctx.handle
    s.rewards, s.values, s.terminals = r.normal(n), r.normal(n), r.chance(n, 1.0 / 60.0)
    s.adv, s.ret = _empty(n), _empty(n)
    return s


def _run_gae(s):
    L.talos_gae(s.ctx, P(s.rewards), P(s.values), P(s.terminals), s.n, 0.99, 0.95, 0.1, 1.3, P(s.adv), P(s.ret))
    L.talos_normalize_slice(s.ctx, P(s.adv), s.n, P(s.adv), None)
    return s.adv, s.ret


def _prepare_dqn(c, seed):
    s, r, ctx = _State(), _Inputs(seed), _ctx()
    n, o, h, a = c["batch"], c["obs"], c["hidden"], c["actions"]
    s.n, s.a, s.mode, s.ctx, s.t = n, a, MODES[c["mode"]], ctx.handle, 0
    dims = [(o, h), (h, h), (h, 1), (h, a)]
    s.layers, at = [], 0        # all parameters in one flat buffer, each matrix on a 16-byte boundary
    for fi, fo in dims:
        w, b = at, at + (fi * fo + 3) // 4 * 4
        s.layers.append((fi, fo, 4 * w, 4 * b))
        at = b + (fo + 3) // 4 * 4
    s.count = at
    s.params, s.grads, s.m, s.v = (torch.zeros(at, device="cuda") for _ in range(4))
    for (fi, fo, w, b) in s.layers:
        s.params[w // 4:w // 4 + fi * fo] = r.xavier(fi, fo).ravel()
    s.target = s.params + r.normal(at, std=0.01) * (s.params != 0)
    s.s0, s.s1, s.actions, s.rewards, s.dones = r.normal(n, o), r.normal(n, o), r.ints(n, a), r.normal(n, std=0.5), r.chance(n, 0.05).float()
    s.nets = {k: [_empty(n, w) for w in (h, h, 1, a, a)] for k in ("now", "next", "frozen")}
    s.tgt, s.loss, s.dq, s.dv, s.da, s.dh2, s.dh1 = _empty(n), _empty(1), _empty(n, a), _empty(n, 1), _empty(n, a), _empty(n, h), _empty(n, h)
    return s


def _run_dqn(s):
    c, n, a, mode = s.ctx, s.n, s.a, s.mode
    none, relu = talos.ACT_NONE, talos.ACT_RELU
    params, grads, target = P(s.params), P(s.grads), P(s.target)
    (o, h, w1, b1), (_, _, w2, b2), (_, _, wv, bv), (_, _, wa, ba) = s.layers

    def q_values(base, x, net):
        h1, h2, v, adv, q = (P(t) for t in net)
        L.talos_linear_fwd(c, P(x), base + w1, base + b1, h1, None, n, o, h, relu, mode)
        L.talos_linear_fwd(c, h1, base + w2, base + b2, h2, None, n, h, h, relu, mode)
        L.talos_linear_fwd(c, h2, base + wv, base + bv, v, None, n, h, 1, none, mode)
        L.talos_linear_fwd(c, h2, base + wa, base + ba, adv, None, n, h, a, none, mode)
        L.talos_dueling_combine_fwd(c, v, adv, q, n, a)
        return q

    q_now = q_values(params, s.s0, s.nets["now"])
    q_next = q_values(params, s.s1, s.nets["next"])
    q_frozen = q_values(target, s.s1, s.nets["frozen"])
    L.talos_dqn_target(c, q_next, q_frozen, P(s.rewards), P(s.dones), 0.99, P(s.tgt), n, a)
    L.talos_dqn_loss_fwd_bwd(c, q_now, P(s.actions), P(s.tgt), P(s.loss), P(s.dq), n, a)
    h1, h2 = P(s.nets["now"][0]), P(s.nets["now"][1])
    dh1, dh2, dv, da = P(s.dh1), P(s.dh2), P(s.dv), P(s.da)
    L.talos_dueling_combine_bwd(c, P(s.dq), dv, da, n, a, 0)
    L.talos_linear_bwd(c, h2, params + wv, None, dv, dh2, grads + wv, grads + bv, n, h, 1, none, mode, 0)
    L.talos_linear_bwd(c, h2, params + wa, None, da, dh2, grads + wa, grads + ba, n, h, a, none, mode, 1)
    L.talos_linear_bwd(c, h1, params + w2, h2, dh2, dh1, grads + w2, grads + b2, n, h, h, relu, mode, 0)
    L.talos_linear_bwd(c, P(s.s0), params + w1, h1, dh1, None, grads + w1, grads + b1, n, o, h, relu, mode, 0)
    s.t += 1
    L.talos_adam_step(c, params, grads, P(s.m), P(s.v), s.count, s.t, 1e-3, 0.9, 0.999, 1e-8, 1.0, 1.0)
    L.talos_soft_update(c, target, params, 0.005, s.count)
    return {"loss": s.loss, "params": s.params, "target": s.target, "grads": s.grads, "m": s.m, "v": s.v}


_KINDS = {k: (globals()["_prepare_" + k], globals()["_run_" + k]) for k in ("update", "rollout", "block", "mla", "mlp", "matmul", "gae", "dqn")}


def prepare(case, seed):
    s = _KINDS[case["kind"]][0](case, seed)
    s.run = _KINDS[case["kind"]][1]
    return s


def run(state):
    return state.run(state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------


def work(case):
    c, k = case, case["kind"]
    if k == "update":
        o, h, a = c["obs"], c["hidden"], c["actions"]
        weights = o * h + h * h + h * (a + 1)
        params = weights + 2 * h + a + 1
        fwd, bwd = 2 * weights, 4 * weights - 2 * o * h         # no gradient with respect to the observations
        passes = c["epochs"] * (fwd + bwd) + (0 if c["host"] else fwd)
        return {"bytes": 4.0 * c["n"] * (o + 4) + 4.0 * params * 2, "flops": float(c["n"]) * passes}
    if k == "rollout":
        n, d, heads, rank, dr = c["sims"], c["hidden"], 4, 32, 16
        weights = 8 * d + d * rank + 2 * rank * d + 2 * d * heads * dr + d * d + d * d + 4 * d * d + d * d + 5 * d
        rows = heads * ((c["context"] + 1) * (2 * d // heads + dr) + (2 * d // heads + dr))      # cached rows read, the new one written
        return {"bytes": 4.0 * (n * (rows + 8 + 5 + 3) + weights), "flops": 2.0 * n * (weights + heads * (c["context"] + 1) * (2 * d // heads + dr))}
    if k == "block":
        t, d, q = c["batch"] * c["seq"], c["width"], c["seq"]
        weights = 4 * d * d + 8 * d * d
        return {"bytes": 4.0 * (4 * t * d + 2 * weights), "flops": 6.0 * t * weights + 2.0 * 6 * t * q * d}
    if k == "mla":
        t, d, r, hd, hr = c["batch"] * c["seq"], c["width"], c["rank"], c["heads"] * c["head"], c["heads"] * c["rope"]
        weights = d * r + 2 * r * hd + d * hd + 2 * d * hr + hd * d
        return {"bytes": 4.0 * (2 * t * d + weights), "flops": 2.0 * t * weights + 2.0 * t * c["seq"] * (2 * hd + hr)}
    if k == "mlp":
        o, h, w = c["obs"], c["hidden"], c["out"]
        weights = o * h + h * h + h * w
        return {"bytes": 4.0 * (c["rows"] * 2 * (o + w) + 2 * weights), "flops": 6.0 * c["rows"] * weights}
    if k == "matmul":
        m, n, q = c["m"], c["n"], c["k"]
        return {"bytes": 8.0 * (m * n + m * q + q * n), "flops": 6.0 * m * n * q}
    if k == "gae":
        return {"bytes": 20.0 * c["n"], "flops": 12.0 * c["n"]}
    o, h, a = c["obs"], c["hidden"], c["actions"]
    weights = o * h + h * h + h * (a + 1)
    return {"bytes": 4.0 * (c["batch"] * (2 * o + 3) + 10 * weights), "flops": 2.0 * c["batch"] * (3 * weights + 2 * weights - o * h)}


def tolerance(case):
    fast = case.get("mode") == "tf32"       # one TF32 product per term: 10 mantissa bits in, fp32 sums
    if case["kind"] in ("update", "dqn"):
        # Adam's step is sign-like where a gradient is at rounding level, so a few weights may move by a learning rate
        # (1 % of the weights' root mean square) each step, however small the difference of the gradients
        return {"rel": 2e-3 if fast else 1e-4, "max": 0.1}
    return {"rel": 2e-3 if fast else 2e-5}
