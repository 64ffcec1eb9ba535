// Linear forward / backward (src/nn.rs:73-133 and the closures it records) as fused GEMM calls.
#include "common.cuh"

namespace {
__global__ void dact_mul_kernel(const float* __restrict__ dy, const float* __restrict__ saved, float* __restrict__ dz,
                                long long n, int act) {
  talos_pdl(dy, saved, dz);
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dz[i] = dy[i] * talos_dact(saved[i], act);
}
// n a multiple of four, 16-byte aligned: two float4 a thread.  SiLU on [65536, 1024] 222 -> 114 us behind the product
// that wrote dY (its three 268 MB streams take 123 us at the measured copy rate; the end of dY is still in L2); one float a
// thread kept too few bytes in flight.
template <int ACT>
__global__ void __launch_bounds__(256)
dact_mul_vec_kernel(const float4* __restrict__ dy, const float4* __restrict__ saved, float4* __restrict__ dz, long long n4) {
  talos_pdl(dy, saved, dz);
  const long long i = (long long)blockIdx.x * 512 + threadIdx.x;
  float4 g[2], s[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) if (i + k * 256 < n4) { g[k] = __ldcs(dy + i + k * 256); s[k] = __ldcs(saved + i + k * 256); }
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (i + k * 256 < n4)
      dz[i + k * 256] = make_float4(g[k].x * talos_dact(s[k].x, ACT), g[k].y * talos_dact(s[k].y, ACT), g[k].z * talos_dact(s[k].z, ACT), g[k].w * talos_dact(s[k].w, ACT));
}
void dact_mul(talos_ctx* ctx, const float* dy, const float* saved, float* dz, int64_t n, int act) {
  if (n % 4 == 0 && (((uintptr_t)dy | (uintptr_t)saved | (uintptr_t)dz) & 15) == 0) {
    auto kern = act == TALOS_ACT_RELU ? dact_mul_vec_kernel<TALOS_ACT_RELU> : act == TALOS_ACT_TANH ? dact_mul_vec_kernel<TALOS_ACT_TANH> : dact_mul_vec_kernel<TALOS_ACT_SILU>;
    talos_kernel(ctx, kern, (unsigned)ceil_div(n / 4, 512), 256, 0, (const float4*)dy, (const float4*)saved, (float4*)dz, n / 4);
  } else {
    talos_kernel(ctx, dact_mul_kernel, (unsigned)ceil_div(n, 256), 256, 0, dy, saved, dz, n, act);
  }
  talos_launched(ctx, "dact_mul");
}
void gemm_any(talos_ctx* ctx, int opA, int opB, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda,
              const float* B, int64_t ldb, float* C, int64_t ldc, int mode, const EpiArgs& e) {
  if (mode != TALOS_MODE_FP32 && talos_gemm_tc_launch(ctx, opA, opB, M, N, K, A, lda, B, ldb, C, ldc, mode, e)) return;
  talos_gemm_fp32_launch(ctx, opA, opB, M, N, K, A, lda, 0, B, ldb, 0, C, ldc, 0, 1, e);
}
}  // namespace

TALOS_API talos_status talos_linear_fwd(talos_ctx* ctx, const float* x, const float* W, const float* bias, float* y,
                                        float* z_save, int64_t rows, int64_t in_f, int64_t out_f, int32_t act,
                                        int32_t mode) {
  TALOS_ENTRY_BEGIN
  talos_check_ctx(ctx);
  TALOS_REQUIRE(rows >= 0 && in_f > 0 && out_f > 0, TALOS_ERR_SHAPE, "MatMul dimension mismatch");
  TALOS_REQUIRE(act >= TALOS_ACT_NONE && act <= TALOS_ACT_SILU && mode >= 0 && mode <= TALOS_MODE_TF32, TALOS_ERR_ARG, "bad act/mode");
  if (rows == 0) return TALOS_OK;
  TALOS_REQUIRE(x && W && y, TALOS_ERR_ARG, "null pointer");
  EpiArgs e{bias, z_save, out_f, nullptr, 0, act, 0, 0};
  gemm_any(ctx, TALOS_OP_N, TALOS_OP_N, rows, out_f, in_f, x, in_f, W, out_f, y, out_f, mode, e);
  TALOS_ENTRY_END
}

TALOS_API talos_status talos_linear_bwd(talos_ctx* ctx, const float* x, const float* W, const float* saved,
                                        const float* dy, float* dx, float* dW, float* db, int64_t rows, int64_t in_f,
                                        int64_t out_f, int32_t act, int32_t mode, int32_t accumulate) {
  TALOS_ENTRY_BEGIN
  talos_check_ctx(ctx);
  TALOS_REQUIRE(rows >= 0 && in_f > 0 && out_f > 0, TALOS_ERR_SHAPE, "MatMul dimension mismatch");
  TALOS_REQUIRE(act >= TALOS_ACT_NONE && act <= TALOS_ACT_SILU && mode >= 0 && mode <= TALOS_MODE_TF32, TALOS_ERR_ARG, "bad act/mode");
  if (rows == 0) return TALOS_OK;
  TALOS_REQUIRE(dy && W && (x || !dW), TALOS_ERR_ARG, "null pointer");
  if (act != TALOS_ACT_NONE) TALOS_REQUIRE(saved != nullptr, TALOS_ERR_ARG, "activation backward needs the saved tensor");
  if (!dx && !dW && !db) return TALOS_OK;
  // Up to 4 096 rows and 2^26 products everything runs as one launch on the CUDA cores: 512 x 64 x 64 with tanh 38 -> 6.5 us in
  // 3xTF32 mode (ten launches before), 1 024 x 256 x 256 56 -> 19 us; beyond that dW's reduction is too long for one
  // cluster and the tensor cores are faster (2 048 x 256 x 256: 36 against 57, 4 096 x 256 x 256: 68 against 59).  A wide layer
  // of few rows, whose dW has more tiles than a round of CTAs, also keeps the separate products: its blocks would be all
  // prologue and store (16 x 2 048 x 2 048 112 us in one launch against 35, 8 x 1 024 x 4 096 200 / 32, 64 x 1 024 x 1 024 59 / 39).  The
  // one launch reads its inputs while it writes its results, so a result that overlaps an input keeps the separate steps, which
  // follow one another: dZ (a copy, where there is an activation, and db with it), dX, dW.
  auto over_input = [&](const float* out, int64_t n) {
    auto hits = [&](const float* p, int64_t m) { return out && p && p < out + n && out < p + m; };
    return hits(dy, rows * out_f) || hits(act ? saved : nullptr, rows * out_f) || hits(x, rows * in_f) || hits(W, in_f * out_f);
  };
  const bool small = rows <= 4096 && rows * in_f * out_f <= (1LL << 26) && !(talos_switches() & SW_TC_NO_SMALL) && !over_input(dx, rows * in_f) &&
                     !over_input(dW, in_f * out_f) && !over_input(db, out_f);
  if (small && (dW || !db) && talos_linear_bwd_small_launch(ctx, x, W, saved, dy, dx, dW, db, rows, in_f, out_f, act, accumulate)) return TALOS_OK;
  // (Up to that size the products stay on the CUDA cores in 3xTF32 mode at 2^26 itself, too: 64 x 2 048 x 512 40 -> 29 us.)
  auto product_mode = [&](int64_t M, int64_t N, int64_t K) {
    return small && mode == TALOS_MODE_TF32X3 && talos_gemm_small_walk(ctx, M, N, K) <= 1024 ? (int32_t)TALOS_MODE_FP32 : mode;
  };
  const float* dz = dy;
  bool db_done = false;
  if (act != TALOS_ACT_NONE) {
    float* buf = (float*)talos_workspace2(ctx, sizeof(float) * (size_t)(rows * out_f));
    // dZ = dY * act'(saved); when the bias gradient is wanted too, the same pass produces its column sums
    if (db && talos_dact_colsum_launch(ctx, dy, buf, saved, act, db, rows, out_f, (accumulate >> 2) & 1)) db_done = true;
    else dact_mul(ctx, dy, saved, buf, rows * out_f, act);
    dz = buf;
  }
  if (dx) {   // dL/dx (+)= dZ . W^T   (src/autograd.rs:275-308)
    EpiArgs e{nullptr, nullptr, 0, nullptr, 0, 0, 0, accumulate & 1};
    gemm_any(ctx, TALOS_OP_N, TALOS_OP_T, rows, in_f, out_f, dz, out_f, W, out_f, dx, in_f, product_mode(rows, in_f, out_f), e);
  }
  if (dW) {   // dL/dW (+)= x^T . dZ   (src/autograd.rs:310-350)
    EpiArgs e{nullptr, nullptr, 0, nullptr, 0, 0, 0, (accumulate >> 1) & 1};
    gemm_any(ctx, TALOS_OP_T, TALOS_OP_N, in_f, out_f, rows, x, in_f, dz, out_f, dW, out_f, product_mode(in_f, out_f, rows), e);
  }
  if (db && !db_done) {   // dL/db (+)= column sums of dZ   (src/autograd.rs:539-543)
    talos_status st = talos_colsum(ctx, dz, db, rows, out_f, (accumulate >> 2) & 1);
    if (st) return st;
  }
  TALOS_ENTRY_END
}
