// The whole optimisation loop of a small policy in one kernel (ppo_small.cu), as the PPO trainer calls it.
#pragma once
#include "common.cuh"

constexpr int PPO_SMALL_MAX = 64;          // widest observation and hidden layer the kernels hold in shared memory
constexpr int PPO_SMALL_HEADS = 32;        // width of the padded heads [policy | value | 0...]

struct PpoSmallNet {                       // flat parameter layout of the trainer
  const float* params; int O, H, A, n_int, o_w1, o_b1, o_w2, o_b2, o_wh, o_bh;
};
struct PpoSmallUpdate {
  PpoSmallNet net;
  const float* obs; const int32_t* actions; const float *old_logp, *adv, *ret;
  long long N; int mb, epochs;             // `epochs` passes over N transitions in consecutive minibatches of mb (the last may be short)
  float *params, *m, *v, *grads;           // grads: the last step's sums and {sum loss, sum kl, count, 0} behind them
  float* stats; int stats_at, stats_slots; // one {sum loss, sum kl, count, 0} per step, from slot stats_at on
  float clip, c_value, c_entropy, lr, b1, b2, eps;
  double b1_t, b2_t;                       // beta1^t and beta2^t of the steps taken before
  int32_t* status;
};
// Largest cluster (16, 8) of the update kernel that the device can place, 0 if none.
int talos_ppo_small_cluster(talos_ctx* ctx);
void talos_ppo_small_update_launch(talos_ctx* ctx, int cluster, const PpoSmallUpdate& a);
// Log-probability of the given actions, or (actions null) logits and values, either of which may be null.
void talos_ppo_small_forward_launch(talos_ctx* ctx, const PpoSmallNet& net, const float* obs, const int32_t* actions, long long N, float* logp, float* logits, float* values);
