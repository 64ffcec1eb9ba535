// fp32 CUDA-core products for small and unaligned problems, in every arithmetic mode: one launch per product (and ONE for
// a whole Linear backward), because at these sizes a launch costs as much as the arithmetic.
//
// What bounds it is latency: a 64 x 64 x 64 product is 0.3 us of arithmetic on four SMs, the rest is the launch and one
// round trip to L2.  So each CTA issues all loads of a 128-deep K chunk at once (two 128-bit loads a thread for either
// operand), the k range of a chunk is shared out over eight (four) groups of warps whose sums meet in shared memory, the
// code a launch walks through is kept short (no divisions, one branch per activation), and a long reduction is split over
// the CTAs of a cluster, which add each other's partial tiles in split order through distributed shared memory (no second
// launch, no trip through L2: partial tiles in global memory and a last-CTA-done counter cost 4 us; the order is fixed, so
// the result is reproducible).
#include "common.cuh"

void talos_splitk_reduce(talos_ctx* ctx, const float* partial, int splits, int64_t M, int64_t N, float* C, int64_t ldc, const EpiArgs& epi);

namespace {

// Reductions longer than this for each CTA of an unslabbed product are cut into slabs.  fp32 mode, x^T.dZ: 64 x 64 x 65 536
// 104 -> 35 us, 64 x 16 x 65 536 60 -> 20, 16 x 16 x 1 048 576 936 -> 75, 256 x 32 x 65 536 106 -> 56, 64 x 256 x 8 192 29 -> 21; at
// 1 024 it is even or slower (64 x 256 x 4 096 16.5 -> 19.1, 64 x 512 x 2 048 18.7 -> 20.6).
constexpr int64_t SLAB_WALK = 1024;

struct SmallOperand {
  const float* p; long long ld, batch;      // element (r, k): p[r*ld + k] when k_contig, else p[k*ld + r]
  const float* saved; int dact;             // multiply every element by act'(saved) at the same index (dact != 0)
  int k_contig;
};
struct SmallProduct {
  SmallOperand a, b;
  float* C; long long ldc, batchC; int vec_c;
  int M, N, K, m_tiles, n_tiles, batch, splits, k_split;    // splits: a power of two; k_split: reduction elements per split, whole chunks
  int k_slab;                               // > 0: batch member z reduces k_slab elements from z * k_slab on (a long reduction in slabs)
  float* colsum; int colsum_acc;            // column sums of B over the whole reduction (the bias gradient), by the m_tile 0 CTAs
  EpiArgs epi;
};

__device__ __forceinline__ float4 dact4(float4 s, int dact) {
  switch (dact) {
    case TALOS_ACT_RELU: return make_float4(talos_dact(s.x, 1), talos_dact(s.y, 1), talos_dact(s.z, 1), talos_dact(s.w, 1));
    case TALOS_ACT_TANH: return make_float4(talos_dact(s.x, 2), talos_dact(s.y, 2), talos_dact(s.z, 2), talos_dact(s.w, 2));
    case TALOS_ACT_SILU: return make_float4(talos_dact(s.x, 3), talos_dact(s.y, 3), talos_dact(s.z, 3), talos_dact(s.w, 3));
    default: return make_float4(1.f, 1.f, 1.f, 1.f);
  }
}
__device__ __forceinline__ float4 act4(float4 v, int act) {
  switch (act) {
    case TALOS_ACT_RELU: return make_float4(talos_act(v.x, 1), talos_act(v.y, 1), talos_act(v.z, 1), talos_act(v.w, 1));
    case TALOS_ACT_TANH: return make_float4(talos_act(v.x, 2), talos_act(v.y, 2), talos_act(v.z, 2), talos_act(v.w, 2));
    case TALOS_ACT_SILU: return make_float4(talos_act(v.x, 3), talos_act(v.y, 3), talos_act(v.z, 3), talos_act(v.w, 3));
    default: return v;
  }
}
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {      // the same shared memory location in CTA `rank` of the cluster
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ld_cluster1(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
// Up to four consecutive floats; `left` of them exist.
__device__ __forceinline__ float4 ld_some(const float* p, int left) {
  float4 v = make_float4(p[0], 0.f, 0.f, 0.f);
  if (left > 1) v.y = p[1];
  if (left > 2) v.z = p[2];
  if (left > 3) v.w = p[3];
  return v;
}
__device__ __forceinline__ void st_some(float* p, float4 v, int left) {
  p[0] = v.x;
  if (left > 1) p[1] = v.y;
  if (left > 2) p[2] = v.z;
  if (left > 3) p[3] = v.w;
}

// One operand's share of a chunk for one thread: LD4 groups of four elements.  Group i covers row r, k .. k+3 (k_contig)
// or rows r .. r+3, k.  The k_contig mapping gives a warp 8 rows x 64 contiguous bytes, so that the scattered stores into
// the k-major tile meet at most two lanes per bank.
template <int R, int KC, int T, int LD4, bool VEC, bool DACT>
struct SmallTile {
  static_assert(R * KC == LD4 * 4 * T, "the threads cover the tile exactly");
  float4 v[LD4];
  static __device__ __forceinline__ void where(bool k_contig, int i, int& r, int& k) {
    if (k_contig) {
      const int blk = (threadIdx.x >> 5) + i * (T / 32), lane = threadIdx.x & 31;
      r = (lane & 7) + 8 * (blk % (R / 8)); k = ((lane >> 3) + 4 * (blk / (R / 8))) * 4;
    } else {
      const int e = threadIdx.x + i * T;
      r = (e % (R / 4)) * 4; k = e / (R / 4);
    }
  }
  __device__ __forceinline__ void load(const SmallOperand& o, long long base, int r0, int rows, int k0, int k_end) {
#pragma unroll
    for (int i = 0; i < LD4; ++i) {
      int r, k; where(o.k_contig, i, r, k);
      r += r0; k += k0;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < rows && k < k_end) {
        const long long off = base + (o.k_contig ? r * o.ld + k : k * o.ld + r);
        const int left = o.k_contig ? k_end - k : rows - r;           // (VEC: the contiguous extent is a multiple of four)
        v[i] = VEC ? *(const float4*)(o.p + off) : ld_some(o.p + off, left);
        if (DACT && o.dact) v[i] = mul4(v[i], dact4(VEC ? *(const float4*)(o.saved + off) : ld_some(o.saved + off, left), o.dact));
      }
    }
  }
  __device__ __forceinline__ void store(bool k_contig, float* s) const {      // s: [KC][R + 4]
#pragma unroll
    for (int i = 0; i < LD4; ++i) {
      int r, k; where(k_contig, i, r, k);
      if (k_contig) {
        s[k * (R + 4) + r] = v[i].x; s[(k + 1) * (R + 4) + r] = v[i].y; s[(k + 2) * (R + 4) + r] = v[i].z; s[(k + 3) * (R + 4) + r] = v[i].w;
      } else {
        *(float4*)(s + k * (R + 4) + r) = v[i];
      }
    }
  }
};

// BM x BN tile, TM x 4 outputs a thread, KG groups of warps that take every KG-th k of a chunk of KC.
template <int BM, int BN, int TM, int KG, int KC>
struct SmallCfg {
  static constexpr int TN = 4, GT = (BM / TM) * (BN / TN), T = GT * KG, PA = BM + 4, PB = BN + 4, BUF = KC * (PA + PB);
  static constexpr int CTAS = T <= 256 ? 3 : BM <= 32 ? 2 : 1;        // resident on an SM at least
  static constexpr int STAGE = 2 * BUF, SUMS = (KG + 1) * BM * BN + T + BN, BYTES = 4 * (STAGE > SUMS ? STAGE : SUMS);   // two chunks, later the groups' sums, column sums and the partial tile
};
template <int BM, int BN, int TM, int KG, int KC, bool VEC, bool DACT>
__device__ __forceinline__ void small_product(const SmallProduct& g, unsigned item, float* sm) {
  using Cfg = SmallCfg<BM, BN, TM, KG, KC>;
  constexpr int TN = Cfg::TN, GT = Cfg::GT, T = Cfg::T, PA = Cfg::PA, PB = Cfg::PB, BUF = Cfg::BUF;
  constexpr int LA = BM * KC / (4 * T), LB = BN * KC / (4 * T), OWN = BM * BN / (4 * T) > 0 ? BM * BN / (4 * T) : 1;
  constexpr bool ALL_OWN = BM * BN >= 4 * T;                // small tile: only the first threads own a float4 of the result
  const int tid = threadIdx.x, kg = tid / GT, tx = (tid % GT) % (BN / TN), ty = (tid % GT) / (BN / TN);
  unsigned mt, nt = 0, bz = 0;
  const unsigned split = item & (unsigned)(g.splits - 1), tile = item >> (31 - __clz(g.splits));
  mt = tile;
  if (tile >= (unsigned)g.m_tiles) { nt = tile / (unsigned)g.m_tiles; mt = tile - nt * (unsigned)g.m_tiles; }
  if (nt >= (unsigned)g.n_tiles) { bz = nt / (unsigned)g.n_tiles; nt -= bz * (unsigned)g.n_tiles; }
  if (bz >= (unsigned)g.batch) {                            // padding of the last cluster: only its barriers
    if (g.splits > 1) { cluster_barrier(); cluster_barrier(); }
    return;
  }
  const int m0 = mt * BM, n0 = nt * BN, k_first = (int)bz * g.k_slab, k_last = g.k_slab ? min(g.K, k_first + g.k_slab) : g.K;
  const int k_begin = min(k_last, k_first + (int)split * g.k_split), k_end = min(k_last, k_begin + g.k_split);
  const long long base_a = bz * g.a.batch, base_b = bz * g.b.batch;
  const bool want_sum = DACT && g.colsum && mt == 0;
  SmallTile<BM, KC, T, LA, VEC, DACT> ta; SmallTile<BN, KC, T, LB, VEC, DACT> tb;
  ta.load(g.a, base_a, m0, g.M, k_begin, k_end); tb.load(g.b, base_b, n0, g.N, k_begin, k_end);
  // this thread's piece of the result; the bias is fetched with the operands, not after the product
  const int own_n = n0 + (tid % (BN / 4)) * 4, own_left = g.N - own_n;
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (g.epi.bias && own_left > 0) bias = ld_some(g.epi.bias + own_n, own_left);
  float acc[TM][TN] = {};
  float csum = 0.f;
  ta.store(g.a.k_contig, sm); tb.store(g.b.k_contig, sm + KC * PA);
  __syncthreads();
  int buf = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += KC) {
    const bool more = k0 + KC < k_end;
    if (more) { ta.load(g.a, base_a, m0, g.M, k0 + KC, k_end); tb.load(g.b, base_b, n0, g.N, k0 + KC, k_end); }
    const float *sa = sm + buf * BUF, *sb = sa + KC * PA;
    const int depth = min(KC, k_end - k0);
#pragma unroll 4
    for (int k = kg; k < depth; k += KG) {
      float a[TM];
#pragma unroll
      for (int i = 0; i + 3 < TM; i += 4) { const float4 q = *(const float4*)(sa + k * PA + ty * TM + i); a[i] = q.x; a[i + 1] = q.y; a[i + 2] = q.z; a[i + 3] = q.w; }
      if (TM == 2) { const float2 q = *(const float2*)(sa + k * PA + ty * TM); a[0] = q.x; a[1] = q.y; }
      const float4 b = *(const float4*)(sb + k * PB + tx * TN);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        acc[i][0] = fmaf(a[i], b.x, acc[i][0]); acc[i][1] = fmaf(a[i], b.y, acc[i][1]);
        acc[i][2] = fmaf(a[i], b.z, acc[i][2]); acc[i][3] = fmaf(a[i], b.w, acc[i][3]);
      }
    }
    if (want_sum) {
#pragma unroll 4
      for (int k = tid / BN; k < depth; k += T / BN) csum += sb[k * PB + tid % BN];
    }
    if (more) { buf ^= 1; ta.store(g.a.k_contig, sm + buf * BUF); tb.store(g.b.k_contig, sm + buf * BUF + KC * PA); }
    __syncthreads();
  }
  // the groups' sums meet in shared memory; each owner thread then adds its float4 in group order
#pragma unroll
  for (int i = 0; i < TM; ++i) *(float4*)(sm + (kg * BM + ty * TM + i) * BN + tx * TN) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  float* const cs = sm + KG * BM * BN;                      // [T / BN][BN]
  if (want_sum) cs[tid] = csum;
  __syncthreads();
  const bool owner = ALL_OWN || tid < BM * BN / 4;
  float4 out[OWN];
#pragma unroll
  for (int j = 0; j < OWN; ++j) {
    out[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (owner) {
#pragma unroll
      for (int q = 0; q < KG; ++q) out[j] = add4(out[j], *(const float4*)(sm + q * BM * BN + (tid + j * T) * 4));
    }
  }
  float col = 0.f;
  if (want_sum && tid < BN) {
#pragma unroll
    for (int q = 0; q < T / BN; ++q) col += cs[q * BN + tid];
  }
  if (g.splits > 1) {
    // every CTA of the tile's group leaves its partial tile in shared memory and adds up its own share of the float4s
    float* const red = sm + Cfg::BYTES / 4 - BM * BN - BN;  // behind the sums being read by slower threads
#pragma unroll
    for (int j = 0; j < OWN; ++j) if (owner) *(float4*)(red + (tid + j * T) * 4) = out[j];
    if (tid < BN) red[BM * BN + tid] = col;
    cluster_barrier();
    uint32_t rank; asm("mov.u32 %0, %cluster_ctarank;" : "=r"(rank));
    const uint32_t first = rank - split;
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
      const bool mine = owner && (unsigned)(tid + j * T) * (unsigned)g.splits / (BM * BN / 4) == split;
      if (mine) {
        out[j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int q = 0; q < g.splits; ++q) out[j] = add4(out[j], ld_cluster4(cluster_addr(red + (tid + j * T) * 4, first + q)));
      }
    }
    if (want_sum && split == 0 && tid < BN) {
      col = 0.f;
      for (int q = 0; q < g.splits; ++q) col += ld_cluster1(cluster_addr(red + BM * BN + tid, first + q));
    }
    cluster_barrier();                                      // nobody leaves while its shared memory may still be read
  }
  float* const C = g.C + bz * g.batchC;
#pragma unroll
  for (int j = 0; j < OWN; ++j) {
    const int m = m0 + (tid + j * T) / (BN / 4);
    if (!owner || m >= g.M || own_left <= 0) continue;
    if (g.splits > 1 && (unsigned)(tid + j * T) * (unsigned)g.splits / (BM * BN / 4) != split) continue;
    float* const c = C + (long long)m * g.ldc + own_n;
    float4 v = add4(out[j], bias);
    if (g.epi.aux_out) st_some(g.epi.aux_out + m * g.epi.ld_aux_out + own_n, v, own_left);
    if (g.epi.act) v = act4(v, g.epi.act);
    if (g.epi.aux_in && g.epi.dact) v = mul4(v, dact4(ld_some(g.epi.aux_in + m * g.epi.ld_aux_in + own_n, own_left), g.epi.dact));
    if (g.epi.beta) v = add4(v, ld_some(c, own_left));
    if (g.vec_c) *(float4*)c = v; else st_some(c, v, own_left);
  }
  if (want_sum && split == 0 && tid < BN && n0 + tid < g.N) g.colsum[n0 + tid] = g.colsum_acc ? g.colsum[n0 + tid] + col : col;
}

template <int BM, int BN, int TM, int KG, int KC, bool VEC>
__global__ void __launch_bounds__((SmallCfg<BM, BN, TM, KG, KC>::T), (SmallCfg<BM, BN, TM, KG, KC>::CTAS))
gemm_small_kernel(const __grid_constant__ SmallProduct g) {
  talos_pdl();
  extern __shared__ __align__(16) float sm[];
  small_product<BM, BN, TM, KG, KC, VEC, false>(g, blockIdx.x, sm);
}
// Linear backward: the first `items_w` CTAs (the longer reductions) work on dW = x^T . dZ and db = column sums of dZ, which
// they have in shared memory anyway, the others on dX = dZ . W^T; dZ = dY * act'(saved) is formed as the tiles are loaded and never
// exists in memory.
template <int BM, int BN, int TM, int KG, int KC, bool VEC>
__global__ void __launch_bounds__((SmallCfg<BM, BN, TM, KG, KC>::T), (BM <= 32 ? 2 : 1))
linear_bwd_small_kernel(const __grid_constant__ SmallProduct gx, const __grid_constant__ SmallProduct gw, unsigned items_w) {
  talos_pdl();
  extern __shared__ __align__(16) float sm[];
  const bool w_role = blockIdx.x < items_w;
  small_product<BM, BN, TM, KG, KC, VEC, true>(w_role ? gw : gx, w_role ? blockIdx.x : blockIdx.x - items_w, sm);
}

int64_t small_tiles(int64_t M, int64_t N, int bm, int bn) { return ceil_div(M, bm) * ceil_div(N, bn); }
bool small_vec(const SmallOperand& o, int64_t rows, int64_t K) {
  return (((uintptr_t)o.p | (uintptr_t)(o.dact ? o.saved : nullptr)) & 15) == 0 && !(o.ld & 3) && !(o.batch & 3) && !((o.k_contig ? K : rows) & 3);
}
// Tiles, and the split of the reduction: as many CTAs as it has chunks while every SM has a slot for them, at most the
// eight of a portable cluster (adding up the partial tiles takes about as long as one chunk).
void small_shape(talos_ctx* ctx, SmallProduct& g, int bm, int bn, int kc, int64_t batch, int64_t slots) {
  g.m_tiles = (int)ceil_div(g.M, bm); g.n_tiles = (int)ceil_div(g.N, bn); g.batch = (int)batch;
  const int64_t tiles = (int64_t)g.m_tiles * g.n_tiles * batch, chunks = std::max<int64_t>(1, ceil_div(g.k_slab ? g.k_slab : g.K, kc));
  int splits = 1;
  while (splits < 8 && splits < chunks && tiles * splits * 2 <= slots) splits *= 2;
  g.splits = splits; g.k_split = (int)(ceil_div(chunks, splits) * kc);
}
int small_tile(talos_ctx* ctx, int64_t tiles16, int64_t tiles32) { return tiles16 <= 2 * ctx->sm_count ? 16 : tiles32 <= 2 * ctx->sm_count ? 32 : 64; }
template <int BM, int BN, int TM, int KG, int KC, bool VEC>
void launch_gemm(talos_ctx* ctx, SmallProduct& g, int64_t batch) {
  using Cfg = SmallCfg<BM, BN, TM, KG, KC>;
  small_shape(ctx, g, BM, BN, KC, batch, Cfg::CTAS * (int64_t)ctx->sm_count);
  static std::atomic<uint64_t> smem_set{0};
  talos_allow_smem(smem_set, (const void*)gemm_small_kernel<BM, BN, TM, KG, KC, VEC>, Cfg::BYTES, ctx->device);
  talos_kernel_cluster(ctx, gemm_small_kernel<BM, BN, TM, KG, KC, VEC>, (unsigned)((int64_t)g.m_tiles * g.n_tiles * batch * g.splits), Cfg::T, Cfg::BYTES, g.splits, g);
}
template <int BM, int TM, int KG, int KC, bool VEC>
void launch_bwd(talos_ctx* ctx, SmallProduct& gx, SmallProduct& gw, int64_t slots) {
  using Cfg = SmallCfg<BM, BM, TM, KG, KC>;
  // How far either reduction is split: the pair that is over first.  A CTA takes its chunks, about two more for its start and its
  // stores and half a one for each doubling of the partial tiles that are added up; past one round of CTAs their work
  // counts, too.  (Leaving dX what dW's split does not take gave dX none: 128 x 512 x 512 28.7 -> 10.9 us.)
  const int64_t tiles_w = gw.C ? small_tiles(gw.M, gw.N, BM, BM) : 0, tiles_x = gx.C ? small_tiles(gx.M, gx.N, BM, BM) : 0;
  const int64_t chunks_w = ceil_div(gw.K, KC), chunks_x = ceil_div(gx.K, KC);
  double best = -1.0;
  for (int sw = 1; sw <= (gw.C ? 8 : 1) && (sw == 1 || sw / 2 < chunks_w); sw *= 2)
    for (int sx = 1; sx <= (gx.C ? 8 : 1) && (sx == 1 || sx / 2 < chunks_x); sx *= 2) {
      const auto taken = [](int64_t chunks, int s) { return (double)ceil_div(chunks, s) + 2.0 + (s == 1 ? 0.0 : s == 2 ? 0.5 : s == 4 ? 1.0 : 1.5); };
      const double cw = tiles_w ? taken(chunks_w, sw) : 0.0, cx = tiles_x ? taken(chunks_x, sx) : 0.0;
      const double cost = std::max(cw, cx) + (tiles_w * sw + tiles_x * sx > slots ? (tiles_w * sw * cw + tiles_x * sx * cx) / (double)slots : 0.0);
      if (best < 0.0 || cost < best) { best = cost; gw.splits = sw; gx.splits = sx; }
    }
  auto shape = [&](SmallProduct& g, int64_t chunks) {
    g.m_tiles = (int)ceil_div(g.M, BM); g.n_tiles = (int)ceil_div(g.N, BM); g.batch = 1; g.k_split = (int)(ceil_div(chunks, g.splits) * KC);
  };
  shape(gw, chunks_w); shape(gx, chunks_x);
  int64_t items_w = tiles_w * gw.splits; const int64_t items_x = tiles_x * gx.splits;
  const int cluster = std::max(gx.splits, gw.splits);
  items_w = ceil_div(items_w, cluster) * cluster;
  static std::atomic<uint64_t> smem_set{0};
  talos_allow_smem(smem_set, (const void*)linear_bwd_small_kernel<BM, BM, TM, KG, KC, VEC>, Cfg::BYTES, ctx->device);
  talos_kernel_cluster(ctx, linear_bwd_small_kernel<BM, BM, TM, KG, KC, VEC>, (unsigned)(items_w + ceil_div(items_x, cluster) * cluster), Cfg::T, Cfg::BYTES, cluster, gx, gw,
                       (unsigned)items_w);
}

// Tile of a product with a long reduction and few tiles: the widest that its result fills, since operands are re-read once
// per tile across them and the slabs keep the SMs busy anyway.
struct SlabTile { int bm, bn, ctas; };
SlabTile slab_tile(int64_t M, int64_t N) {
  if (M > 32 && N > 32) return {64, 64, SmallCfg<64, 64, 4, 1, 32>::CTAS};
  if (M > 16 && N <= 16) return {64, 16, SmallCfg<64, 16, 4, 4, 64>::CTAS};
  if (M > 16) return {32, 32, SmallCfg<32, 32, 4, 8, 128>::CTAS};
  return {16, 16, SmallCfg<16, 16, 2, 16, 128>::CTAS};
}

}  // namespace

// Reduction elements one CTA walks for a plain product on these kernels.
int64_t talos_gemm_small_walk(talos_ctx* ctx, int64_t M, int64_t N, int64_t K) {
  const int tile = small_tile(ctx, small_tiles(M, N, 16, 16), small_tiles(M, N, 32, 32));
  const int64_t tiles = small_tiles(M, N, tile, tile), slots = (tile == 64 ? 1 : 2) * (int64_t)ctx->sm_count, chunks = ceil_div(K, tile == 64 ? 64 : 128);
  int64_t splits = 1;
  while (splits < 8 && splits < chunks && tiles * splits * 2 <= slots) splits *= 2;
  return ceil_div(K, splits);
}

// C = op(A).op(B) with the epilogue, any shape and alignment.
void talos_gemm_small_launch(talos_ctx* ctx, int opA, int opB, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, int64_t strideA, const float* B,
                             int64_t ldb, int64_t strideB, float* C, int64_t ldc, int64_t strideC, int64_t batch, const EpiArgs& epi) {
  SmallProduct g{};
  g.a = SmallOperand{A, lda, batch > 1 ? strideA : 0, nullptr, 0, opA == TALOS_OP_N};
  g.b = SmallOperand{B, ldb, batch > 1 ? strideB : 0, nullptr, 0, opB == TALOS_OP_T};
  g.C = C; g.ldc = ldc; g.batchC = batch > 1 ? strideC : 0; g.M = (int)M; g.N = (int)N; g.K = (int)K; g.epi = epi;
  g.vec_c = !(((uintptr_t)C) & 15) && !(ldc & 3) && !(g.batchC & 3) && !(N & 3);
  const bool vec = small_vec(g.a, M, K) && small_vec(g.b, N, K);
  // The tile is the smallest that leaves the product in one round of CTAs (two of the smaller ones fit an SM): an SM's fp32 units
  // take 1 024 cycles for a chunk of a 32 x 32 tile and a quarter of that for a 16 x 16 one, which is what is left once
  // the launch and the loads are as short as they get; larger tiles re-read the operands less often.
#define TALOS_SMALL(BM, BN, TM, KG, KC) { if (vec) launch_gemm<BM, BN, TM, KG, KC, true>(ctx, g, batch); else launch_gemm<BM, BN, TM, KG, KC, false>(ctx, g, batch); }
  // Few tiles and a long reduction (a first layer's weight gradient over a large fp32 minibatch): a cluster's eight CTAs would
  // walk it alone, so it is cut into slabs, a cluster each, as many as fill the SMs; their results go through memory.
  if (batch == 1 && K > SLAB_WALK && talos_gemm_small_walk(ctx, M, N, K) > SLAB_WALK) {
    const SlabTile t = slab_tile(M, N);
    // as many clusters as there are slots, or fewer where the SMs then share them more evenly
    const int64_t tiles = small_tiles(M, N, t.bm, t.bn), sms = ctx->sm_count, most = t.ctas * sms / (8 * tiles);
    auto filled = [&](int64_t slabs) { const int64_t ctas = 8 * tiles * slabs; return (double)ctas / (double)(ceil_div(ctas, sms) * sms); };
    int64_t even = most;
    for (int64_t s = most; s > 0 && 2 * s >= most; --s) if (filled(s) > filled(even) + 0.01) even = s;
    const int64_t want = std::min(even, K / 1024);
    if (want > 1) {
      g.k_slab = (int)(ceil_div(ceil_div(K, want), 128) * 128);       // whole chunks: the vector loads stay aligned
      batch = ceil_div(K, g.k_slab);
      g.C = (float*)talos_workspace(ctx, sizeof(float) * (size_t)(batch * M * N)); g.ldc = N; g.batchC = M * N; g.vec_c = !(N & 3); g.epi = EpiArgs{};
      if (t.bm == 16) TALOS_SMALL(16, 16, 2, 16, 128) else if (t.bm == 32) TALOS_SMALL(32, 32, 4, 8, 128) else if (t.bn == 16) TALOS_SMALL(64, 16, 4, 4, 64)
      else TALOS_SMALL(64, 64, 4, 1, 32)
      talos_launched(ctx, "gemm_small");
      talos_splitk_reduce(ctx, g.C, (int)batch, M, N, C, ldc, epi);
      return;
    }
  }
  // Past one round, three CTAs of 256 threads an SM hide each other's loads and stores: a narrow result (a head's logits) takes
  // 64 x 16 tiles (65 536 x 5 x 64: 31 -> 13 us, 20 000 x 5 x 64: 13.5 -> 5.9), a short reduction tiles whose k range is not
  // shared out, since those sums cost more than 64 products do (65 536 x 64 x 8: 18 -> 9.1 us, 8 192 x 256 x 16: 11.3 -> 7.4; within
  // one round the shared-out range stays ahead, 1 200 x 256 x 64: 5.4 against 8.6, and so do 32 x 32 tiles, 8 192 x 16 x 256: 9.7
  // against 11.3).
  const bool in_place = talos_result_over_operand(opA, opB, M, N, K, A, lda, strideA, B, ldb, strideB, C, ldc, strideC, batch, epi);
  const int tile = in_place ? 64 : small_tile(ctx, ceil_div(M, 16) * ceil_div(N, 16) * batch, ceil_div(M, 32) * ceil_div(N, 32) * batch);
  const bool rounds = ceil_div(M, 64) * ceil_div(N, 64) * batch > ctx->sm_count;
  if (tile == 16) TALOS_SMALL(16, 16, 2, 16, 128) else if (tile == 32) TALOS_SMALL(32, 32, 4, 8, 128) else if (N <= 16) TALOS_SMALL(64, 16, 4, 4, 64)
  else if (K <= 64 && rounds) TALOS_SMALL(64, 64, 4, 1, 32) else TALOS_SMALL(64, 64, 8, 4, 64)
#undef TALOS_SMALL
  talos_launched(ctx, "gemm_small");
}

// dX (+)= dZ.W^T, dW (+)= x^T.dZ, db (+)= column sums of dZ, dZ = dY * act'(saved), in one launch (dx or dW/db may be null;
// db comes with dW).  False, nothing launched: dW alone has more tiles than a round of CTAs.
bool talos_linear_bwd_small_launch(talos_ctx* ctx, const float* x, const float* W, const float* saved, const float* dy, float* dx, float* dW, float* db,
                                   int64_t rows, int64_t in_f, int64_t out_f, int act, int accumulate) {
  const int tile = small_tile(ctx, (dx ? small_tiles(rows, in_f, 16, 16) : 0) + (dW ? small_tiles(in_f, out_f, 16, 16) : 0),
                              (dx ? small_tiles(rows, in_f, 32, 32) : 0) + (dW ? small_tiles(in_f, out_f, 32, 32) : 0));
  const int64_t slots = (tile == 64 ? 1 : 2) * (int64_t)ctx->sm_count;
  if (dW && small_tiles(in_f, out_f, tile, tile) > slots) return false;
  SmallProduct gx{}, gw{};
  bool vec = true;
  if (dx) {
    gx.a = SmallOperand{dy, out_f, 0, saved, act, 1}; gx.b = SmallOperand{W, out_f, 0, nullptr, 0, 1};
    gx.C = dx; gx.ldc = in_f; gx.M = (int)rows; gx.N = (int)in_f; gx.K = (int)out_f; gx.epi.beta = accumulate & 1;
    gx.vec_c = !(((uintptr_t)dx) & 15) && !(in_f & 3);
    vec = vec && small_vec(gx.a, rows, out_f) && small_vec(gx.b, in_f, out_f);
  }
  if (dW) {
    gw.a = SmallOperand{x, in_f, 0, nullptr, 0, 0}; gw.b = SmallOperand{dy, out_f, 0, saved, act, 0};
    gw.C = dW; gw.ldc = out_f; gw.M = (int)in_f; gw.N = (int)out_f; gw.K = (int)rows; gw.epi.beta = (accumulate >> 1) & 1;
    gw.vec_c = !(((uintptr_t)dW) & 15) && !(out_f & 3); gw.colsum = db; gw.colsum_acc = (accumulate >> 2) & 1;
    vec = vec && small_vec(gw.a, in_f, rows) && small_vec(gw.b, out_f, rows);
  }
#define TALOS_SMALL(BM, TM, KG, KC) { if (vec) launch_bwd<BM, TM, KG, KC, true>(ctx, gx, gw, slots); else launch_bwd<BM, TM, KG, KC, false>(ctx, gx, gw, slots); }
  if (tile == 16) TALOS_SMALL(16, 2, 16, 128) else if (tile == 32) TALOS_SMALL(32, 4, 8, 128) else TALOS_SMALL(64, 8, 4, 64)
#undef TALOS_SMALL
  talos_launched(ctx, "linear_bwd_small");
  return true;
}
