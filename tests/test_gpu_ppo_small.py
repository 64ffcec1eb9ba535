"""The one-launch update and forward of small policies (ppo_small.cu) where their loops end: minibatches below and around the
16 CTAs x 16 rows of a block, ragged last minibatches, widths up to 64 and 31 actions, odd widths (padding of the flat layout),
lane groups of 8, 16 and 32 per row, all arithmetic modes (they share the kernel).  The reference is the float64 oracle;
fp32 sums of at most 4 096 terms keep a gradient within 1e-5 of it in the 2-norm (sqrt(4096) * 2^-23 = 8e-6 for the longest)."""
import numpy as np
import pytest

from oracle import model as om
import oracle as orc
from gpu_util import dev, host, rel_err
from test_gpu_ppo import make_problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(talos):
    c = talos.torch_context(0)
    yield c
    c.synchronize()


@pytest.mark.parametrize("N,mb,O,H,A,mode", [(1, 1, 8, 64, 5, 1), (15, 64, 8, 64, 5, 0), (257, 256, 1, 64, 7, 1), (300, 64, 64, 64, 31, 1), (520, 260, 12, 33, 8, 2),
                                             (1000, 2048, 16, 64, 15, 1), (2049, 2049, 16, 64, 15, 1), (2048, 272, 8, 64, 16, 1), (900, 300, 7, 5, 1, 0)])
def test_gradients_and_weights(talos, ctx, N, mb, O, H, A, mode):
    obs, actions, adv, ret, params = make_problem(N, O, H, A, seed=200)
    for k in ("b1", "b2", "bp", "bv"):
        params[k] = orc.f32r(orc.rng_normal(211, params[k].shape, 0.0, 0.1))
    model = om.MlpActorCritic(params)
    old = orc.f32r(model.log_prob(obs, actions) + orc.rng_normal(210, (N,), 0.0, 0.2))          # ratios on both sides of the clip
    tr = talos.PPOTrainer(ctx, talos.PpoConfig(O, H, A, mb, mode, lr=1e-3)); tr.set_params(params)
    d = [dev(x) for x in (obs, actions, old, adv, ret)]
    import torch
    lp = torch.empty(N, device="cuda"); tr.log_prob(d[0], d[1], N, lp)
    assert np.abs(host(lp) - model.log_prob(obs, actions)).max() <= 1e-5
    # one minibatch: every gradient, the loss, one launch
    n = min(N, mb)
    tr.step(*[x[:n].contiguous() for x in d], n)
    g_ref, loss_ref, _ = model.grads(obs[:n], actions[:n], old[:n], adv[:n], ret[:n])
    got = tr.get_grads()
    for k in g_ref:
        assert rel_err(got[k], g_ref[k]) <= 1e-5, (k, rel_err(got[k], g_ref[k]))
    assert (tr.launches_per_step == 1) == (mb <= 2048)
    # all minibatches of two epochs, the optimizer's state carried on from that step
    tr.set_params(params); tr.reset_optimizer()
    kls = tr.update(*d, N, 2, 0.0)
    ref_kls, _ = om.ppo_update(model, obs, actions, old, adv, ret, 2, mb, lr=np.float64(np.float32(1e-3)), kl_stop=None)
    assert np.allclose(kls, ref_kls, rtol=1e-3, atol=1e-6)
    weights = tr.get_params()
    for k in weights:
        assert rel_err(weights[k], model.p[k]) <= (1e-5 if k.startswith("w") else 1e-3), (k, rel_err(weights[k], model.p[k]))
    # host-staged and early-stopping forms run epoch by epoch, the arithmetic is the same
    for form in (dict(host=True), dict(kl_stop=1e9)):
        tr.set_params(params); tr.reset_optimizer()
        args = [np.ascontiguousarray(host(x).astype(np.int32 if x.dtype == torch.int32 else np.float32)) for x in d] if "host" in form else d
        tr.update(*args, N, 2, **form)
        again = tr.get_params()
        assert all(np.array_equal(again[k], weights[k]) for k in weights)
    tr.close()


def test_an_unknown_action_is_reported(talos, ctx):
    import torch
    obs, actions, adv, ret, params = make_problem(64, 8, 64, 5, seed=220)
    actions = actions.copy(); actions[40] = 5
    tr = talos.PPOTrainer(ctx, talos.PpoConfig(8, 64, 5, 32, 1)); tr.set_params(params)
    d_obs, d_act, z = dev(obs), dev(actions), torch.zeros(64, device="cuda")
    with pytest.raises(Exception):
        tr.update(d_obs, d_act, z, dev(adv), dev(ret), 64, 1, 0.0)
    out = torch.empty(64, device="cuda")
    tr.log_prob(d_obs, d_act, 64, out)
    with pytest.raises(Exception):
        ctx.synchronize()
    ctx.synchronize()
    tr.close()


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_one_forward_with_and_without_a_communicator(talos, ctx, mode):
    # The log-probabilities stored before an update and those of its first step, taken with a communicator (of one rank), come from
    # the same arithmetic.  Logits of about 30: fp32 rounding puts 1e-5 into a log-ratio and 2^-24 into (ratio - 1) - log(ratio); TF32
    # on one side would put 1e-2 into the log-ratio and 1e-4 into the KL.
    import torch
    n = 512
    obs, actions, adv, ret, params = make_problem(n, 8, 64, 5, seed=230)
    params["wp"] = orc.f32r(params["wp"] * 12.0)
    comm = talos.Comm(ctx, talos.Comm.unique_id(), 1, 0)
    tr = talos.PPOTrainer(ctx, talos.PpoConfig(8, 64, 5, n, mode), comm); tr.set_params(params)
    d_obs, d_act, old = dev(obs), dev(actions), torch.empty(n, device="cuda")
    tr.log_prob(d_obs, d_act, n, old)
    kls = tr.update(d_obs, d_act, old, dev(adv), dev(ret), n, 1, 0.0)
    assert abs(kls[0]) <= 1e-6, kls
    tr.close(); comm.close()
