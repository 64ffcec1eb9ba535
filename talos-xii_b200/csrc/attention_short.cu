// Attention over short sequences (S <= 128, heads of at most 64), forward with saved probabilities and backward from them, one
// launch each, one CTA a head.
//
// What bounds it is memory: a head of 64 x 32 is 0.4 MFLOP on 24 KB of operands and 16 KB of probabilities.  As three
// (forward) and five (backward) launches over batched products the scores crossed HBM six and eleven times, and a 128-row
// tensor-core tile is half padding at S = 64.  Here a head's operands are read once into shared memory, the scores live in registers
// (thread (ty, tx) of 16 x 16 holds rows ty + 16 i and columns tx + 16 j, so that a row's maximum and sum are shuffles
// within half a warp) and only the probabilities are written.  The fp32 units take every arithmetic mode: no less precise than the
// mode asks for.  Rows are padded to 16 DC + 4 floats, an odd number of 128-bit words, and zero past the head's width and the
// sequence's end, so that no product has a special case.  (8 192 heads of 64 x 32 take 211 us forward and 330 us backward, 61 and 91 us
// by their bytes: shared-memory reads are what is left, three 128-bit loads for every sixteen products' issue slots.)
#include <algorithm>
#include <initializer_list>

#include "common.cuh"

namespace {

constexpr int AT = 256;

template <int TS, int DC> struct ShortCfg {
  static constexpr int M = TS / 16, PD = 16 * DC + 4, PS = TS + 4, HEAD = TS * PD, PROB = TS * PS;
  static constexpr int FWD = 4 * (3 * HEAD + PROB), BWD = 4 * (4 * HEAD + PROB);
  static constexpr int CTAS = M == 8 ? 1 : 3;             // resident at least: bounds the registers
};

__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) {
  acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc); acc = fmaf(a.z, b.z, acc); return fmaf(a.w, b.w, acc);
}
template <int N> struct Vec;                              // N consecutive floats
template <> struct Vec<1> { using T = float; };
template <> struct Vec<2> { using T = float2; };
template <> struct Vec<4> { using T = float4; };
template <int N> __device__ __forceinline__ void ld_vec(float (&d)[N], const float* p) { *(typename Vec<N>::T*)d = *(const typename Vec<N>::T*)p; }
template <int N> __device__ __forceinline__ void st_vec(float* p, const float (&s)[N]) { *(typename Vec<N>::T*)p = *(const typename Vec<N>::T*)s; }

// A head [S][d] into [TS][PD], zero elsewhere; magic divides by d / 4.
template <int TS, int PD>
__device__ __forceinline__ void load_head(float* s, const float* g, int S, int d, unsigned magic) {
  const int d4 = d >> 2;
  for (int c = threadIdx.x; c < S * d4; c += AT) {
    const int r = (int)__umulhi((unsigned)c, magic);
    *(float4*)(s + r * PD + (c - r * d4) * 4) = ((const float4*)g)[c];
  }
  constexpr int W = PD / 4;                               // the padding columns and rows
  if (S < TS || d4 < W) {
    for (int c = threadIdx.x; c < TS * W; c += AT) {
      const int r = c / W, q = c % W;
      if (r >= S || q >= d4) *(float4*)(s + r * PD + 4 * q) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}
// acc[i][j] = row ty + 16 i of a . row tx + 16 j of b; column blocks above the diagonal are left out when `causal`.
template <int M, int DC, int PD>
__device__ __forceinline__ void scores(float (&acc)[M][M], const float* a, const float* b, int ty, int tx, int d, int causal) {
#pragma unroll
  for (int i = 0; i < M; ++i)
#pragma unroll
    for (int j = 0; j < M; ++j) acc[i][j] = 0.f;
  for (int c = 0; c < d; c += 4) {
    float4 x[M];
#pragma unroll
    for (int i = 0; i < M; ++i) x[i] = *(const float4*)(a + (ty + 16 * i) * PD + c);
#pragma unroll
    for (int j = 0; j < M; ++j) {
      const float4 y = *(const float4*)(b + (tx + 16 * j) * PD + c);
#pragma unroll
      for (int i = 0; i < M; ++i) if (!causal || j <= i) acc[i][j] = dot4(x[i], y, acc[i][j]);
    }
  }
}
// out[row][col] = sum over c of p[row][c] . b[c][col]: rows ty + 16 i, columns tx DC .. tx DC + DC - 1.
template <int M, int DC, int PD, int PS>
__device__ __forceinline__ void rows_by_head(const float* p, const float* b, float* out, int ty, int tx, int S, int d) {
  float acc[M][DC] = {};
#pragma unroll 2
  for (int c = 0; c < S; c += 4) {
    float y[4][DC];
#pragma unroll
    for (int e = 0; e < 4; ++e) ld_vec<DC>(y[e], b + (c + e) * PD + tx * DC);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      const float4 x = *(const float4*)(p + (ty + 16 * i) * PS + c);
#pragma unroll
      for (int j = 0; j < DC; ++j) {
        acc[i][j] = fmaf(x.x, y[0][j], acc[i][j]); acc[i][j] = fmaf(x.y, y[1][j], acc[i][j]);
        acc[i][j] = fmaf(x.z, y[2][j], acc[i][j]); acc[i][j] = fmaf(x.w, y[3][j], acc[i][j]);
      }
    }
  }
  if (tx * DC >= d) return;
#pragma unroll
  for (int i = 0; i < M; ++i) if (ty + 16 * i < S) st_vec<DC>(out + (size_t)(ty + 16 * i) * d + tx * DC, acc[i]);
}
// out[col][d] = sum over rows r of p[r][col] . b[r][d]: columns M ty .. M ty + M - 1 of p.
template <int M, int DC, int PD, int PS>
__device__ __forceinline__ void columns_by_head(const float* p, const float* b, float* out, int ty, int tx, int S, int d) {
  float acc[M][DC] = {};
#pragma unroll 4
  for (int r = 0; r < S; ++r) {
    float x[M], y[DC];
    constexpr int V = M < 4 ? M : 4;
#pragma unroll
    for (int i = 0; i < M; i += V) ld_vec<V>(*(float(*)[V])(x + i), p + r * PS + M * ty + i);
    ld_vec<DC>(y, b + r * PD + tx * DC);
#pragma unroll
    for (int i = 0; i < M; ++i)
#pragma unroll
      for (int j = 0; j < DC; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
  }
  if (tx * DC >= d) return;
#pragma unroll
  for (int i = 0; i < M; ++i) if (M * ty + i < S) st_vec<DC>(out + (size_t)(M * ty + i) * d + tx * DC, acc[i]);
}
__device__ __forceinline__ float half_max(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float half_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int TS, int DC>
__global__ void __launch_bounds__(AT, (ShortCfg<TS, DC>::CTAS))
attention_short_fwd_kernel(const float* q, const float* k, const float* v, float* out, float* probs, int S, int dqk, int dv, unsigned magic_qk, unsigned magic_v,
                           float scale, int causal) {
  talos_pdl(q, k, v, out, probs);
  using Cfg = ShortCfg<TS, DC>;
  constexpr int M = Cfg::M, PD = Cfg::PD, PS = Cfg::PS;
  extern __shared__ __align__(16) float sm[];
  float *const Q = sm, *const K = Q + Cfg::HEAD, *const V = K + Cfg::HEAD, *const Pm = V + Cfg::HEAD;
  const size_t bh = blockIdx.x;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  load_head<TS, PD>(Q, q + bh * S * dqk, S, dqk, magic_qk);
  load_head<TS, PD>(K, k + bh * S * dqk, S, dqk, magic_qk);
  load_head<TS, PD>(V, v + bh * S * dv, S, dv, magic_v);
  __syncthreads();
  float s[M][M];
  scores<M, DC, PD>(s, Q, K, ty, tx, dqk, causal);
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const int r = ty + 16 * i, lim = causal ? min(r + 1, S) : S;
    float mx = -INFINITY, sum = 0.f;
#pragma unroll
    for (int j = 0; j < M; ++j) { s[i][j] *= scale; if (tx + 16 * j < lim) mx = fmaxf(mx, s[i][j]); }
    mx = half_max(mx);
#pragma unroll
    for (int j = 0; j < M; ++j) { s[i][j] = tx + 16 * j < lim ? expf(s[i][j] - mx) : 0.f; sum += s[i][j]; }
    const float inv = 1.f / half_sum(sum);
#pragma unroll
    for (int j = 0; j < M; ++j) {
      const int c = tx + 16 * j;
      const float p = s[i][j] * inv;
      Pm[r * PS + c] = p;
      if (probs && r < S && c < S) probs[(bh * S + r) * S + c] = p;
    }
  }
  __syncthreads();
  rows_by_head<M, DC, PD, PS>(Pm, V, out + bh * S * dv, ty, tx, S, dv);
}

// dV = P^T.dO ; dP = dO.V^T ; dS = scale * P * (dP - rowsum(dP * P)) ; dQ = dS.K ; dK = dS^T.Q
template <int TS, int DC>
__global__ void __launch_bounds__(AT, (ShortCfg<TS, DC>::CTAS))
attention_short_bwd_kernel(const float* q, const float* k, const float* v, const float* probs, const float* dout, float* dq, float* dk, float* dv, int S, int dqk, int dvd,
                           unsigned magic_qk, unsigned magic_v, float scale) {
  talos_pdl(q, k, v, probs, dout, dq, dk, dv);
  using Cfg = ShortCfg<TS, DC>;
  constexpr int M = Cfg::M, PD = Cfg::PD, PS = Cfg::PS;
  extern __shared__ __align__(16) float sm[];
  float *const Q = sm, *const K = Q + Cfg::HEAD, *const V = K + Cfg::HEAD, *const dO = V + Cfg::HEAD, *const Pm = dO + Cfg::HEAD;
  const size_t bh = blockIdx.x;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float p[M][M], s[M][M];
#pragma unroll
  for (int i = 0; i < M; ++i)
#pragma unroll
    for (int j = 0; j < M; ++j) {
      const int r = ty + 16 * i, c = tx + 16 * j;
      p[i][j] = r < S && c < S ? probs[(bh * S + r) * S + c] : 0.f;
    }
  load_head<TS, PD>(V, v + bh * S * dvd, S, dvd, magic_v);
  load_head<TS, PD>(dO, dout + bh * S * dvd, S, dvd, magic_v);
  load_head<TS, PD>(Q, q + bh * S * dqk, S, dqk, magic_qk);
  load_head<TS, PD>(K, k + bh * S * dqk, S, dqk, magic_qk);
#pragma unroll
  for (int i = 0; i < M; ++i)
#pragma unroll
    for (int j = 0; j < M; ++j) Pm[(ty + 16 * i) * PS + tx + 16 * j] = p[i][j];
  __syncthreads();
  columns_by_head<M, DC, PD, PS>(Pm, dO, dv + bh * S * dvd, ty, tx, S, dvd);
  scores<M, DC, PD>(s, dO, V, ty, tx, dvd, 0);
  __syncthreads();                                        // everybody is done with P; dS takes its place
#pragma unroll
  for (int i = 0; i < M; ++i) {
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < M; ++j) dot = fmaf(s[i][j], p[i][j], dot);
    dot = half_sum(dot);
#pragma unroll
    for (int j = 0; j < M; ++j) Pm[(ty + 16 * i) * PS + tx + 16 * j] = scale * (p[i][j] * (s[i][j] - dot));
  }
  __syncthreads();
  rows_by_head<M, DC, PD, PS>(Pm, K, dq + bh * S * dqk, ty, tx, S, dqk);
  columns_by_head<M, DC, PD, PS>(Pm, Q, dk + bh * S * dqk, ty, tx, S, dqk);
}

unsigned magic4(int64_t d) { const uint64_t d4 = (uint64_t)d / 4; return (unsigned)(((uint64_t(1) << 32) + d4 - 1) / d4); }     // exact below 2^32 / d4

template <int TS, int DC>
void launch_fwd(talos_ctx* ctx, const float* q, const float* k, const float* v, float* out, float* probs, int64_t BH, int S, int dqk, int dv, float scale, int causal) {
  static std::atomic<uint64_t> smem_set{0};
  talos_allow_smem(smem_set, (const void*)attention_short_fwd_kernel<TS, DC>, ShortCfg<TS, DC>::FWD, ctx->device);
  talos_kernel(ctx, attention_short_fwd_kernel<TS, DC>, (unsigned)BH, AT, ShortCfg<TS, DC>::FWD, q, k, v, out, probs, S, dqk, dv, magic4(dqk), magic4(dv), scale, causal);
  talos_launched(ctx, "attention_short_fwd");
}
template <int TS, int DC>
void launch_bwd(talos_ctx* ctx, const float* q, const float* k, const float* v, const float* probs, const float* dout, float* dq, float* dk, float* dv, int64_t BH, int S, int dqk,
                int dvd, float scale) {
  static std::atomic<uint64_t> smem_set{0};
  talos_allow_smem(smem_set, (const void*)attention_short_bwd_kernel<TS, DC>, ShortCfg<TS, DC>::BWD, ctx->device);
  talos_kernel(ctx, attention_short_bwd_kernel<TS, DC>, (unsigned)BH, AT, ShortCfg<TS, DC>::BWD, q, k, v, probs, dout, dq, dk, dv, S, dqk, dvd, magic4(dqk), magic4(dvd), scale);
  talos_launched(ctx, "attention_short_bwd");
}

}  // namespace

// What the tiles hold, in whole 128-bit pieces (at least two a row) -- and where this is the faster route.  In fp32 mode it always is
// (8 192 heads of 64 x 32, causal: forward 772 -> 212 us, backward 667 -> 330; 4 096 of 128 x 64: 2 056 -> 874, 1 674 -> 1 291).  The
// tensor-core products take over when their 128-row tiles are full and the head is wide enough (3xTF32, forward / backward: 64 x 32
// 269 -> 211 / 496 -> 330 us, 50 x 64 529 -> 305 / 809 -> 566, but 64 x 64 314 against 330 / 593 against 626, 96 x 32 226 against 465 /
// 385 against 627).  Before that counts there must be more heads than SMs: one round of CTAs is over before the products'
// three and five launches are (96 heads of 128 x 32, 3xTF32: 22 -> 17 / 37 -> 24 us; only TF32's backward of 64-wide heads is not:
// 33 against 37).  They also refuse batches whose rows are not whole 128-bit words (S % 4), which then went to the fp32 kernels.
bool talos_attention_short_takes(talos_ctx* ctx, int64_t BH, int64_t S, int64_t dqk, int64_t dv, int mode, std::initializer_list<const void*> heads) {
  uintptr_t bits = 0;
  for (const void* p : heads) bits |= (uintptr_t)p;
  if (!(BH < (int64_t(1) << 31) && S >= 1 && S <= 128 && dqk >= 8 && dv >= 8 && dqk <= 64 && dv <= 64 && dqk % 4 == 0 && dv % 4 == 0 && (bits & 15) == 0)) return false;
  const bool wide = std::max(dqk, dv) > 32;
  if (mode == TALOS_MODE_FP32 || S % 4 != 0 || (S <= 64 && (S <= 48 || !wide))) return true;
  return BH <= ctx->sm_count && !(mode == TALOS_MODE_TF32 && S > 64 && wide);
}
#define TALOS_SHORT(F, WIDTH, ...)                                                                                               \
  {                                                                                                                             \
    const int64_t w = WIDTH;                                                                                                    \
    if (S <= 32) { if (w <= 16) F<32, 1>(__VA_ARGS__); else if (w <= 32) F<32, 2>(__VA_ARGS__); else F<32, 4>(__VA_ARGS__); }    \
    else if (S <= 64) { if (w <= 16) F<64, 1>(__VA_ARGS__); else if (w <= 32) F<64, 2>(__VA_ARGS__); else F<64, 4>(__VA_ARGS__); } \
    else { if (w <= 16) F<128, 1>(__VA_ARGS__); else if (w <= 32) F<128, 2>(__VA_ARGS__); else F<128, 4>(__VA_ARGS__); }         \
  }
void talos_attention_short_fwd(talos_ctx* ctx, const float* q, const float* k, const float* v, float* out, float* probs, int64_t BH, int64_t S, int64_t dqk, int64_t dv,
                               float scale, int causal) {
  TALOS_SHORT(launch_fwd, std::max(dqk, dv), ctx, q, k, v, out, probs, BH, (int)S, (int)dqk, (int)dv, scale, causal)
}
void talos_attention_short_bwd(talos_ctx* ctx, const float* q, const float* k, const float* v, const float* probs, const float* dout, float* dq, float* dk, float* dv, int64_t BH,
                               int64_t S, int64_t dqk, int64_t dvd, float scale) {
  TALOS_SHORT(launch_bwd, std::max(dqk, dvd), ctx, q, k, v, probs, dout, dq, dk, dv, BH, (int)S, (int)dqk, (int)dvd, scale)
}
#undef TALOS_SHORT
