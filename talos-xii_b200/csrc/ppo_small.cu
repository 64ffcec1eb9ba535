// Policies of at most 64 observations, 64 hidden units and 31 actions, in small minibatches (the reference's own settings are 8, 64, 5
// and 256): every minibatch of every epoch in ONE launch of one thread-block cluster.
//
// What bounds such an update is the chain of dependent steps, each a few microseconds of arithmetic: eleven launches a step
// took 84 us (2 048 transitions, 8 epochs of minibatch 256: 5.4 ms; now 9.2 us a step, 0.66 ms).  Here the weights live in the shared memory of each of
// the cluster's 16 CTAs, a CTA takes its share of the minibatch in blocks of 16 rows through forward, loss and backward
// without leaving shared memory, and the gradient sums meet through distributed shared memory: each parameter has one owner
// thread in the cluster, which adds the CTAs' sums in rank order (the result does not depend on timing), keeps
// the Adam moments in registers and stores the new weight into every CTA.  Two cluster barriers a step, no trip
// through L2 but for the transitions, which are fetched a block ahead.
//
// Products run on the fp32 units in every arithmetic mode: 16 x 64 x 64 is 512 cycles of an SM's FMA rate, less than a tensor-core
// tile needs to be set up and read back, and no less precise than the mode asks for.  Operands are laid out so that a
// thread's 4 x 4 outputs cost two 128-bit loads per reduction element (rows of activations contiguous: [unit][row]); the
// reduction is shared by four (heads: eight) groups of threads whose partial sums meet in shared memory in group order.
#include "ppo_small.cuh"

namespace {

constexpr int T = 256, RB = 16, U = PPO_SMALL_MAX, HP = PPO_SMALL_HEADS;
constexpr int PR = RB + 4, PW = U + 4, PH = HP + 4;       // pitches: eight 128-bit accesses a phase meet all banks
constexpr int G_MAX = 2 * (U * U + U) + U * HP + HP;      // most parameters (every section is a multiple of four)

struct Net {                                              // shared memory: weights, activations of one block of rows, partial sums
  float w1[U * PW], w2[U * PW], wh[U * PH], b1[U], b2[U], bh[HP];
  float x[U * PR], h1[U * PR], h2[U * PR], z[HP * PR], part[8 * RB * PH];
};
static_assert(8 * RB * PH >= 4 * RB * PW, "the partial sums of both groupings fit");
struct Train : Net {
  float dh1[U * PR], dh2[U * PR], g[G_MAX + 4], rows[4 * RB], loss[RB], kl[RB], inv_bc[4];
};

__device__ __forceinline__ float4 ld4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ void fma16(float (&acc)[4][4], float4 a, float4 b) {
  const float x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
}
__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) {
  acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc); acc = fmaf(a.z, b.z, acc); return fmaf(a.w, b.w, acc);
}

// Partial products part[group][row][column] of a[k][row] (activations) and w[k][column]; GROUPS groups of T / GROUPS threads
// take every GROUPS-th k.  Columns: 4 T / GROUPS / 4 = 64 (four groups) or 32 (eight).
template <int GROUPS, int P>
__device__ __forceinline__ void product(const float* a, const float* w, int K, float* part) {
  constexpr int GT = T / GROUPS, CG = GT / 4;             // threads of a group, column groups
  const int g = threadIdx.x / GT, rg = (threadIdx.x % GT) / CG, cg = threadIdx.x % CG;
  float acc[4][4] = {};
#pragma unroll 4
  for (int k = g; k < K; k += GROUPS) fma16(acc, ld4(a + k * PR + 4 * rg), ld4(w + k * P + 4 * cg));
#pragma unroll
  for (int i = 0; i < 4; ++i) *(float4*)(part + (g * RB + 4 * rg + i) * P + 4 * cg) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}
// The same with the transposed weights, w[column][k]: a thread's columns are 16 apart so that its 128-bit reads along k of
// eight neighbouring columns meet all banks.  K counts whole groups of four.
template <int P>
__device__ __forceinline__ void product_t(const float* a, const float* w, int K4, float* part) {
  const int g = threadIdx.x >> 6, rg = (threadIdx.x & 63) >> 4, cg = threadIdx.x & 15;
  float acc[4][4] = {};
  for (int q = g; q < K4; q += 4) {
    float4 y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = ld4(w + (cg + 16 * j) * P + 4 * q);
#define TALOS_STEP(e, c) fma16(acc, ld4(a + (4 * q + e) * PR + 4 * rg), make_float4(y[0].c, y[1].c, y[2].c, y[3].c));
    TALOS_STEP(0, x) TALOS_STEP(1, y) TALOS_STEP(2, z) TALOS_STEP(3, w)
#undef TALOS_STEP
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) part[(g * RB + 4 * rg + i) * PW + cg + 16 * j] = acc[i][j];
}
// The four groups' sums of this thread's unit and four rows.
__device__ __forceinline__ float4 sum_parts(const float* part) {
  const int c = threadIdx.x & 63, r = (threadIdx.x >> 6) * 4;
  float s[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float* p = part + (r + i) * PW + c;
    s[i] = ((p[0] + p[RB * PW]) + p[2 * RB * PW]) + p[3 * RB * PW];
  }
  return make_float4(s[0], s[1], s[2], s[3]);
}
__device__ __forceinline__ void finish_tanh(const float* part, const float* bias, float* h, int H) {
  const int c = threadIdx.x & 63, r = (threadIdx.x >> 6) * 4;
  float4 s = sum_parts(part);
  const float b = bias[c];
  s = c < H ? make_float4(talos_tanh(s.x + b), talos_tanh(s.y + b), talos_tanh(s.z + b), talos_tanh(s.w + b)) : make_float4(0.f, 0.f, 0.f, 0.f);
  *(float4*)(h + c * PR + r) = s;
}
__device__ __forceinline__ void finish_dtanh(const float* part, const float* h, float* dh) {
  const int c = threadIdx.x & 63, r = (threadIdx.x >> 6) * 4;
  const float4 s = sum_parts(part), y = ld4(h + c * PR + r);
  *(float4*)(dh + c * PR + r) = make_float4(s.x * (1.f - y.x * y.x), s.y * (1.f - y.y * y.y), s.z * (1.f - y.z * y.z), s.w * (1.f - y.w * y.w));
}
// x [unit][row] -> h1, h2, z; ends with a barrier, z complete.
__device__ __forceinline__ void forward(Net* s, int O, int H, int A) {
  product<4, PW>(s->x, s->w1, O, s->part); __syncthreads();
  finish_tanh(s->part, s->b1, s->h1, H); __syncthreads();
  product<4, PW>(s->h1, s->w2, H, s->part); __syncthreads();
  finish_tanh(s->part, s->b2, s->h2, H); __syncthreads();
  product<8, PH>(s->h2, s->wh, H, s->part); __syncthreads();
  const int c = threadIdx.x & 31, r = (threadIdx.x >> 5) * 2;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    float v = 0.f;
#pragma unroll
    for (int g = 0; g < 8; ++g) v += s->part[(g * RB + r + i) * PH + c];
    s->z[c * PR + r + i] = c <= A ? v + s->bh[c] : 0.f;
  }
  __syncthreads();
}
// Where parameter e of the flat layout lies in shared memory, as a float index into Net; -1 for the layout's padding.
__device__ __forceinline__ int weight_at(const PpoSmallNet& n, int e) {
  const Net* s = nullptr;
  const auto at = [&](const float* base, int i) { return (int)(base - (const float*)s) + i; };
  if (e >= n.o_bh) return e - n.o_bh < HP ? at(s->bh, e - n.o_bh) : -1;
  if (e >= n.o_wh) { const int i = e - n.o_wh; return i < n.H * HP ? at(s->wh, i / HP * PH + i % HP) : -1; }
  if (e >= n.o_b2) { const int i = e - n.o_b2; return i < n.H ? at(s->b2, i) : -1; }
  if (e >= n.o_w2) { const int i = e - n.o_w2; return i < n.H * n.H ? at(s->w2, i / n.H * PW + i % n.H) : -1; }
  if (e >= n.o_b1) { const int i = e - n.o_b1; return i < n.H ? at(s->b1, i) : -1; }
  return e < n.O * n.H ? at(s->w1, e / n.H * PW + e % n.H) : -1;
}
// All weights (zero where the network is narrower than the arrays); the caller's next barrier publishes them.
__device__ __forceinline__ void load_weights(Net* s, const PpoSmallNet& n) {
  constexpr int W = 2 * U * PW + U * PH + 2 * U + HP;
  for (int i = threadIdx.x; i < W; i += T) ((float*)s)[i] = 0.f;
  __syncthreads();
#pragma unroll 8
  for (int e = threadIdx.x; e < n.n_int; e += T) {
    const int at = weight_at(n, e);
    const float w = n.params[e];
    if (at >= 0) ((float*)s)[at] = w;
  }
}
// This thread's elements of a block of observations: rows row0 .. row0 + valid - 1, zero behind them.
struct Rows {
  float x[4]; int at[4];                                  // at: places in the [unit][row] array, -1 past the block
  __device__ __forceinline__ explicit Rows(int O) {
#pragma unroll
    for (int j = 0; j < 4; ++j) { const int i = threadIdx.x + T * j; at[j] = i < RB * O ? i % O * PR + i / O : -1; }
  }
  __device__ __forceinline__ void load(const float* obs, long long row0, int valid, int O) {
#pragma unroll
    for (int j = 0; j < 4; ++j) { const int i = threadIdx.x + T * j; x[j] = i < valid * O ? obs[row0 * O + i] : 0.f; }
  }
  __device__ __forceinline__ void store(float* xs) const {
#pragma unroll
    for (int j = 0; j < 4; ++j) if (at[j] >= 0) xs[at[j]] = x[j];
  }
};
// Lanes that share a row of the heads: the power of two that holds A logits and the value.
__device__ __forceinline__ int lanes_per_row(int A) { return A < 8 ? 8 : A < 16 ? 16 : 32; }
template <bool MAX>
__device__ __forceinline__ float lane_reduce(float v, int width) {
  for (int o = width >> 1; o > 0; o >>= 1) { const float w = __shfl_xor_sync(0xffffffffu, v, o); v = MAX ? fmaxf(v, w) : v + w; }
  return v;
}

__device__ __forceinline__ void cluster_barrier() { asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float ld_cluster(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(uint32_t a, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }

// Where a CTA is in its walk over epochs, minibatches and its 16-row blocks of each.
struct Walk {
  int epoch, block; long long first; int n, share, lo;
  __device__ __forceinline__ void open(const PpoSmallUpdate& a, int C, int rank) {
    n = (int)min((long long)a.mb, a.N - first); share = (n + C - 1) / C; lo = rank * share; block = 0;
  }
  __device__ __forceinline__ int valid() const { return max(0, min(RB, min(share, n - lo) - block * RB)); }
  __device__ __forceinline__ long long row0() const { return first + lo + block * RB; }
  __device__ __forceinline__ bool last_block() const { return (block + 1) * RB >= share; }
  __device__ __forceinline__ void next(const PpoSmallUpdate& a, int C, int rank) {
    if (!last_block()) { ++block; return; }
    first += a.mb;
    if (first >= a.N) { first = 0; ++epoch; }
    open(a, C, rank);
  }
};

template <int C>
__global__ void __launch_bounds__(T, 1)
ppo_small_update_kernel(const __grid_constant__ PpoSmallUpdate a) {
  talos_pdl();
  extern __shared__ __align__(16) float sm[];
  Train* const s = (Train*)sm;
  const int tid = threadIdx.x, O = a.net.O, H = a.net.H, A = a.net.A, n_int = a.net.n_int;
  const int rank = (int)blockIdx.x;                       // the grid is one cluster
  load_weights(s, a.net);
  for (int i = tid; i < G_MAX + 4; i += T) s->g[i] = 0.f;
  if (tid < RB) { s->loss[tid] = 0.f; s->kl[tid] = 0.f; }
  // the parameters this thread owns
  constexpr int OWN = (G_MAX + 4 + C * T - 1) / (C * T);
  float p[OWN], m[OWN], v[OWN]; int at[OWN];
#pragma unroll
  for (int j = 0; j < OWN; ++j) {
    const int e = (j * C + rank) * T + tid;
    at[j] = e < n_int ? weight_at(a.net, e) : -1;
    p[j] = m[j] = v[j] = 0.f;
    if (at[j] >= 0) { p[j] = a.params[e]; m[j] = a.m[e]; v[j] = a.v[e]; }
  }
  double b1_t = a.b1_t, b2_t = a.b2_t;                    // (thread T - 1 only)
  Walk w{}; w.open(a, C, rank);
  Rows xr(O); float rv = 0.f;                                // the next block's observations, and its (action, old log-prob, advantage, return)
  const auto fetch = [&](const Walk& k) {
    if (k.epoch >= a.epochs) return;
    const int valid = k.valid(), r = tid & (RB - 1);
    xr.load(a.obs, k.row0(), valid, O);
    rv = 0.f;
    if (tid < 4 * RB && r < valid) {
      const float* src = tid < RB ? (const float*)a.actions : tid < 2 * RB ? a.old_logp : tid < 3 * RB ? a.adv : a.ret;
      rv = src[k.row0() + r];
    }
  };
  fetch(w);
  const int kg = tid >> 4, cg = tid & 15;                 // weight-gradient outputs: units kg + 16 i by columns cg + 16 j
  const int LW = lanes_per_row(A);
  cluster_barrier();                                      // every CTA's weights are in place before anybody stores new ones there
  for (int step = 0; w.epoch < a.epochs; ++step) {
    float dw1[4][4] = {}, dw2[4][4] = {}, dwh[4][2] = {}, db = 0.f;
    const int n = w.n;
    bool more = true;
    while (more) {
      const int valid = w.valid();
      more = !w.last_block();
      if (tid == T - 1 && !more) {                        // Adam's bias corrections of this step
        b1_t *= (double)a.b1; b2_t *= (double)a.b2;
        s->inv_bc[0] = (float)(1.0 / (1.0 - b1_t)); s->inv_bc[1] = (float)(1.0 / (1.0 - b2_t));
      }
      if (valid > 0) {
        xr.store(s->x);
        if (tid < 4 * RB) s->rows[tid] = rv;
      }
      w.next(a, C, rank);
      fetch(w);
      if (valid == 0) continue;                           // uniform in the CTA
      __syncthreads();
      forward(s, O, H, A);
      // loss and its gradient with respect to [logits | value], LW lanes a row (the per-sample graph of src/ppo.rs:702-755)
      for (int r = tid / LW; r < RB; r += T / LW) {
        const int c = tid & (LW - 1), act = __float_as_int(s->rows[r]);
        const float old = s->rows[RB + r], advantage = s->rows[2 * RB + r], ret = s->rows[3 * RB + r];
        const float l = c < A ? s->z[c * PR + r] : -INFINITY, value = s->z[A * PR + r];
        const float mx = lane_reduce<true>(l, LW);
        const float lse = logf(lane_reduce<false>(c < A ? expf(l - mx) : 0.f, LW)) + mx;
        const float lp = c < A ? l - lse : 0.f, pr = c < A ? expf(lp) : 0.f;
        const float ent = -lane_reduce<false>(pr * lp, LW);
        const bool known = act >= 0 && act < A;
        float lp_a = __shfl_sync(0xffffffffu, lp, ((tid & 31) & ~(LW - 1)) + (known ? act : 0));
        if (!known) lp_a = 0.f;                           // reported; the sample contributes its entropy and value terms only
        const float log_ratio = lp_a - old, ratio = expf(log_ratio), kl = (ratio - 1.f) - log_ratio;
        const float lo = 1.f - a.clip, hi = 1.f + a.clip;
        const float surr1 = ratio * advantage, surr2 = fminf(fmaxf(ratio, lo), hi) * advantage;
        const bool use1 = surr1 < surr2;
        const float d_ratio = use1 ? advantage : ((ratio >= lo && ratio <= hi) ? advantage : 0.f);
        const float dvl = value - ret;
        const float d = c < A ? a.c_entropy * pr * (lp + 1.f) + (c == act ? -(d_ratio * ratio) : 0.f) : 0.f;
        const float sum_d = lane_reduce<false>(d, LW);
        float out = c < A ? d - pr * sum_d : c == A ? a.c_value * 2.f * dvl : 0.f;
        if (r >= valid) out = 0.f;
        __syncwarp();                                     // the row's value has been read by all its lanes
        s->z[c * PR + r] = out;
        if (c == 0 && r < valid) {
          if (!known) atomicExch(a.status, TALOS_DEV_BAD_INDEX);
          s->loss[r] += -(use1 ? surr1 : surr2) + a.c_value * dvl * dvl - a.c_entropy * ent; s->kl[r] += kl;
        }
      }
      __syncthreads();
      product_t<PH>(s->z, s->wh, (A + 4) >> 2, s->part); __syncthreads();
      finish_dtanh(s->part, s->h2, s->dh2); __syncthreads();
      product_t<PW>(s->dh2, s->w2, (H + 3) >> 2, s->part);
      for (int r = 0; r < RB; r += 4) {
        float4 y[4], q[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) { y[j] = ld4(s->dh2 + (cg + 16 * j) * PR + r); q[j] = ld4(s->h1 + (kg + 16 * j) * PR + r); }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) dw2[i][j] = dot4(q[i], y[j], dw2[i][j]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (16 * j > A) continue;
          const float4 dz = ld4(s->z + (cg + 16 * j) * PR + r);
#pragma unroll
          for (int i = 0; i < 4; ++i) dwh[i][j] = dot4(ld4(s->h2 + (kg + 16 * i) * PR + r), dz, dwh[i][j]);
        }
      }
      __syncthreads();
      finish_dtanh(s->part, s->h1, s->dh1); __syncthreads();
      for (int r = 0; r < RB; r += 4) {
        float4 y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = ld4(s->dh1 + (cg + 16 * j) * PR + r);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (16 * i >= O) continue;
          const float4 q = ld4(s->x + (kg + 16 * i) * PR + r);
#pragma unroll
          for (int j = 0; j < 4; ++j) dw1[i][j] = dot4(q, y[j], dw1[i][j]);
        }
      }
      if (tid < 2 * U + HP) {
        const float* d = tid < U ? s->dh1 + tid * PR : tid < 2 * U ? s->dh2 + (tid - U) * PR : s->z + (tid - 2 * U) * PR;
        const float4 q0 = ld4(d), q1 = ld4(d + 4), q2 = ld4(d + 8), q3 = ld4(d + 12);
        db += (((q0.x + q0.y) + (q0.z + q0.w)) + ((q1.x + q1.y) + (q1.z + q1.w))) + (((q2.x + q2.y) + (q2.z + q2.w)) + ((q3.x + q3.y) + (q3.z + q3.w)));
      }
      __syncthreads();                                    // the block's arrays are free
    }
    // this CTA's sums, in the flat layout
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = kg + 16 * i;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = cg + 16 * j;
        if (k < O && c < H) s->g[a.net.o_w1 + k * H + c] = dw1[i][j];
        if (k < H && c < H) s->g[a.net.o_w2 + k * H + c] = dw2[i][j];
        if (j < 2 && k < H) s->g[a.net.o_wh + k * HP + c] = dwh[i][j < 2 ? j : 0];
      }
    }
    if (tid < U) { if (tid < H) s->g[a.net.o_b1 + tid] = db; }
    else if (tid < 2 * U) { if (tid - U < H) s->g[a.net.o_b2 + tid - U] = db; }
    else if (tid < 2 * U + HP) s->g[a.net.o_bh + tid - 2 * U] = db;
    else if (tid < 2 * U + HP + 2) {
      float* const part = tid == 2 * U + HP ? s->loss : s->kl;
      float t = 0.f;
      for (int r = 0; r < RB; ++r) { t += part[r]; part[r] = 0.f; }
      s->g[n_int + tid - 2 * U - HP] = t;
    }
    cluster_barrier();
    float g[OWN];
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
      const int e = (j * C + rank) * T + tid;
      g[j] = 0.f;
      if (e < n_int + 2) {
#pragma unroll
        for (int q = 0; q < C; ++q) g[j] += ld_cluster(cluster_addr(s->g + e, q));
      }
    }
    const float coef = 1.f / fmaxf((float)n, 1.f), inv_bc1 = s->inv_bc[0], inv_bc2 = s->inv_bc[1];
    const bool final_step = w.epoch >= a.epochs;
    float* const stats = a.stats + 4 * (size_t)((a.stats_at + step) % a.stats_slots);
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
      const int e = (j * C + rank) * T + tid;
      if (at[j] >= 0) {                                   // Adam::step (src/ppo.rs:519-533)
        const float gi = g[j] * coef;
        m[j] = a.b1 * m[j] + (1.f - a.b1) * gi; v[j] = a.b2 * v[j] + (1.f - a.b2) * gi * gi;
        p[j] -= a.lr * (m[j] * inv_bc1) / (sqrtf(v[j] * inv_bc2) + a.eps);
#pragma unroll
        for (int q = 0; q < C; ++q) st_cluster(cluster_addr((float*)s + at[j], q), p[j]);
      }
      if (e >= n_int && e < n_int + 4) stats[e - n_int] = e == n_int + 2 ? (float)n : g[j];
      if (final_step && e < n_int + 4) {
        a.grads[e] = e == n_int + 2 ? (float)n : g[j];
        if (at[j] >= 0) { a.params[e] = p[j]; a.m[e] = m[j]; a.v[e] = v[j]; }
      }
    }
    cluster_barrier();                                    // the new weights are everywhere, and nobody reads the sums any more
  }
}

__global__ void __launch_bounds__(T, 2)
ppo_small_forward_kernel(PpoSmallNet net, const float* obs, const int32_t* actions, long long N, float* logp, float* logits, float* values, int32_t* status) {
  talos_pdl(net.params, obs, actions, logp, logits, values, status);
  extern __shared__ __align__(16) float sm[];
  Net* const s = (Net*)sm;
  const int tid = threadIdx.x, A = net.A, LW = lanes_per_row(A);
  Rows xr(net.O);
  long long row0 = (long long)blockIdx.x * RB;
  xr.load(obs, row0, (int)min((long long)RB, N - row0), net.O);
  load_weights(s, net);
  for (; row0 < N; row0 += (long long)gridDim.x * RB) {
    const int valid = (int)min((long long)RB, N - row0);
    xr.store(s->x);
    const long long next = row0 + (long long)gridDim.x * RB;
    if (next < N) xr.load(obs, next, (int)min((long long)RB, N - next), net.O);
    __syncthreads();
    forward(s, net.O, net.H, A);
    for (int r = tid / LW; r < RB; r += T / LW) {
      const int c = tid & (LW - 1);
      const float l = c < A ? s->z[c * PR + r] : -INFINITY;
      if (logp) {
        const float mx = lane_reduce<true>(l, LW);
        const float lse = logf(lane_reduce<false>(c < A ? expf(l - mx) : 0.f, LW)) + mx;
        if (c == 0 && r < valid) {
          const int act = actions[row0 + r];
          if (act < 0 || act >= A) { atomicExch(status, TALOS_DEV_BAD_INDEX); logp[row0 + r] = 0.f; }    // no read outside the row; reported at the next sync
          else logp[row0 + r] = s->z[act * PR + r] - lse;
        }
      } else if (r < valid) {
        if (c < A && logits) logits[(row0 + r) * A + c] = l;
        if (c == A && values) values[row0 + r] = s->z[A * PR + r];
      }
    }
    __syncthreads();
  }
}

template <int C>
int cluster_fits(talos_ctx* ctx) {
  const void* const kern = (const void*)ppo_small_update_kernel<C>;
  if (C > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) { cudaGetLastError(); return 0; }
  static std::atomic<uint64_t> smem_set{0};
  talos_allow_smem(smem_set, kern, sizeof(Train), ctx->device);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = C; cfg.blockDim = T; cfg.dynamicSmemBytes = sizeof(Train); cfg.stream = ctx->stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension; attr.val.clusterDim.x = C; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
  cfg.attrs = &attr; cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
  return clusters > 0 ? C : 0;
}

}  // namespace

int talos_ppo_small_cluster(talos_ctx* ctx) {
  const int c = cluster_fits<16>(ctx);
  return c ? c : cluster_fits<8>(ctx);
}
void talos_ppo_small_update_launch(talos_ctx* ctx, int cluster, const PpoSmallUpdate& a) {
  if (cluster == 16) talos_kernel_cluster(ctx, ppo_small_update_kernel<16>, 16, T, sizeof(Train), 16, a);
  else talos_kernel_cluster(ctx, ppo_small_update_kernel<8>, 8, T, sizeof(Train), 8, a);
  talos_launched(ctx, "ppo_small_update");
}
void talos_ppo_small_forward_launch(talos_ctx* ctx, const PpoSmallNet& net, const float* obs, const int32_t* actions, long long N, float* logp, float* logits, float* values) {
  if (N == 0) return;
  static std::atomic<uint64_t> smem_set{0};
  talos_allow_smem(smem_set, (const void*)ppo_small_forward_kernel, sizeof(Net), ctx->device);
  const unsigned grid = (unsigned)std::min<int64_t>(ceil_div(N, RB), 2 * (int64_t)ctx->sm_count);      // two CTAs fit an SM
  talos_kernel(ctx, ppo_small_forward_kernel, grid, T, sizeof(Net), net, obs, actions, N, logp, logits, values, ctx->dev_status);
  talos_launched(ctx, "ppo_small_forward");
}
