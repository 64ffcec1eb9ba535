// Shared host-side plumbing for the talos_b200 library: context, error reporting, launch checks.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>
#include <stdexcept>
#include <string>

#include "../../include/talos_b200.h"

#define TALOS_API extern "C" __attribute__((visibility("default")))

struct talos_error : std::runtime_error {
  talos_status code;
  talos_error(talos_status c, const std::string& m) : std::runtime_error(m), code(c) {}
};

void talos_set_last_error(const std::string& msg);

// (The runtime keeps a failed call's error for cudaGetLastError, too: taken here, or the next launch would report it again.)
#define TALOS_CHECK_CUDA(expr)                                                                     \
  do {                                                                                             \
    cudaError_t e__ = (expr);                                                                      \
    if (e__ != cudaSuccess) {                                                                      \
      (void)cudaGetLastError();                                                                    \
      throw talos_error(TALOS_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e__));      \
    }                                                                                              \
  } while (0)

#define TALOS_REQUIRE(cond, code, msg)                                                             \
  do {                                                                                             \
    if (!(cond)) throw talos_error((code), std::string(msg) + " [" #cond "]");                     \
  } while (0)

// Wraps the body of every extern "C" entry point: exceptions become status codes.
#define TALOS_ENTRY_BEGIN try {
#define TALOS_ENTRY_END                                                                            \
  return TALOS_OK;                                                                                 \
  }                                                                                                \
  catch (const talos_error& e) { talos_set_last_error(e.what()); return e.code; }                  \
  catch (const std::bad_alloc&) { talos_set_last_error("host allocation failed"); return TALOS_ERR_ALLOC; } \
  catch (const std::exception& e) { talos_set_last_error(e.what()); return TALOS_ERR_CUDA; }

struct talos_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int sm_count = 148;
  void* ws = nullptr;          // kernel-level scratch: split-K partials, column-sum / reduction partials
  size_t ws_bytes = 0;
  void* ws2 = nullptr;         // op-level scratch of composite entry points: dZ of Linear backward, dS of attention
  size_t ws2_bytes = 0;
  int32_t* dev_status = nullptr;   // device-side error word: 1000..2999 a bounded wait gave up, 3000 an index argument was out of range
  int32_t* host_status = nullptr;  // pinned host copy, refreshed by every entry point that blocks on the stream
  int tc_state = 0;            // tensor-core GEMM: 0 = not probed, 1 = active, -1 = disabled
  std::atomic<int64_t> launches{0};
  unsigned dbg_wait_spins = 0;     // test hook (talos_debug_gemm_stall): poll limit of the GEMM kernels' bounded waits, 0 = default
  int dbg_skip_kb = -1;            // test hook: k-block the first CTA's loader leaves out, -1 = none
  struct talos_pool* pool = nullptr;   // caching device allocator behind talos_malloc / talos_free (ctx.cu)
  struct talos_timeline* timeline = nullptr;   // measurement aid (talos_ctx_timeline_begin): one event per launch while recording
};
// Records an event behind the launch just made (ctx.cu); only called while a timeline is being recorded.
void talos_timeline_mark(talos_ctx* ctx, const char* what);

// Device-side error codes written to talos_ctx::dev_status (first writer wins is not required: any non-zero value reports).
#define TALOS_DEV_TIMEOUT_BASE 1000    // + CTA index % 1000 (+ 1000 from the CTA-pair kernel): a bounded mbarrier / flag wait gave up  -> TALOS_ERR_TIMEOUT
#define TALOS_DEV_BAD_INDEX 3000       // an action / index argument read from device memory was out of range -> TALOS_ERR_ARG

// Blocks until the ctx stream is idle, then reports (and clears) the device-side error word: every entry point that
// already waits for the stream calls this instead of cudaStreamSynchronize, so a kernel that gave up is never followed
// by a silent TALOS_OK.
void talos_sync_and_check(talos_ctx* ctx);
// Looks up the device address of talos_colsum_noalloc's fixed scratch array for `device` (which must be current).
void talos_colsum_noalloc_prepare(int device);

// Returns a scratch pointer of at least `bytes`, growing the buffer (stream-ordered free of the
// old one) when needed.
void* talos_workspace(talos_ctx* ctx, size_t bytes);
// Same for the op-level scratch.  Composite entry points use this one so that the kernels they
// call can take their own partial-sum scratch from talos_workspace without overlapping it.
void* talos_workspace2(talos_ctx* ctx, size_t bytes);

inline void talos_check_ctx(talos_ctx* ctx) {
  TALOS_REQUIRE(ctx != nullptr, TALOS_ERR_ARG, "null context");
  TALOS_CHECK_CUDA(cudaSetDevice(ctx->device));
}

// Programmatic dependent launch.  Every kernel of the library calls talos_pdl() before it touches memory: its CTAs may be
// set up while the kernel before it on the stream is still running (its launch, its CTAs' set-up and its code fetch then
// overlap that kernel's tail), they read and write nothing before griddepcontrol.wait has seen that kernel complete, and they
// let the next kernel be set up in turn.  It is the first statement but in the tensor-memory kernels, which call it behind the
// block barrier that publishes their allocation: the call of any one thread lets the next kernel start, and two waiting
// kernels' CTAs must not compete for an SM's columns (the later one would hold them and wait for the earlier one to
// complete, the earlier one would wait for the columns).  The launch itself is cheaper, too: 2.07 -> 1.55 us of host time each, and a chain of tiny
// dependent kernels takes 1.6 us a link instead of 2.1 (B200, driver 580).
// The kernel's pointers are passed through it because a load that the compiler knows to be read-only (__restrict__ const, __ldg,
// __ldcs) may otherwise be moved above the wait; kernels that take their pointers in a struct use plain loads, or send the
// pointer through such a barrier where they use it (the forward epilogue's bias: as a plain load it cost 3 us of a 364 us step).
template <typename... T>
__device__ __forceinline__ void talos_pdl(T&... ptrs) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  ((void)([&] { asm volatile("" : "+l"(ptrs) : : "memory"); }()), ...);
}
// Launches `kern` (which must call talos_pdl() as said above) on the ctx stream, `cluster` CTAs to a cluster.  Follow it with talos_launched.
template <typename... P, typename... A>
inline void talos_kernel_cluster(talos_ctx* ctx, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, unsigned cluster, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension; attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 2 : 1;
  TALOS_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
}
template <typename... P, typename... A>
inline void talos_kernel(talos_ctx* ctx, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
  talos_kernel_cluster(ctx, kern, grid, block, smem, 1u, args...);
}

// Call after every kernel launch.
inline void talos_launched(talos_ctx* ctx, const char* what) {
  ctx->launches.fetch_add(1, std::memory_order_relaxed);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) throw talos_error(TALOS_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
  if (ctx->timeline) talos_timeline_mark(ctx, what);
}

// The measurement switches (environment variables TALOS_*) that are set right now, as a bit mask: ONE walk over the
// environment per call instead of one per switch (a dozen getenv calls were 1.5 us of every tensor-core launch).
enum : unsigned {
  SW_DISABLE_TENSOR_CORES = 1u << 0, SW_TC_NO_SHORTK = 1u << 1, SW_TC_NO_WIDE_EPI = 1u << 2, SW_TC_NO_EARLY = 1u << 3, SW_TC_NO_PREFETCH = 1u << 4,
  SW_TC_FORCE_PAIR = 1u << 5, SW_TC_NO_PAIR = 1u << 6, SW_TC_NO_RASTER = 1u << 7, SW_TC_NO_FOLD = 1u << 8, SW_TC_NO_FUSED_DACT = 1u << 9,
  SW_TC_NO_EPI8 = 1u << 10, SW_ATTN_NO_FUSED = 1u << 11, SW_TC_NO_SMALL = 1u << 12
};
unsigned talos_switches();
// Raises a kernel's dynamic shared memory limit once per device (`done`: one bit per device, a static of the launcher).
inline void talos_allow_smem(std::atomic<uint64_t>& done, const void* kern, size_t bytes, int device) {
  const uint64_t bit = 1ull << (device & 63);
  if (device < 64 && (done.load(std::memory_order_acquire) & bit)) return;
  TALOS_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  done.fetch_or(bit, std::memory_order_release);
}

static inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// ---- activation helpers shared by the GEMM epilogues and the elementwise kernels ----
// tanh(x) = 1 - 2 / (2^(2x log2 e) + 1) with the hardware exp2 / reciprocal approximations: five dependent
// instructions, no branch, correct limits (+-1) without clamping, |abs error| < 3e-7 (the GEMM epilogues are
// instruction-latency bound, so the short chain matters more than the last bit near zero, where the RELATIVE
// error of this form grows as 1e-7 / |x|).
__device__ __forceinline__ float talos_tanh(float x) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * 2.8853900817779268f));   // exp(2x) = 2^(2x log2 e)
  return 1.f - __fdividef(2.f, e + 1.f);                                         // 2/inf = 0 and 2/1 give the +-1 limits
}
__device__ __forceinline__ float talos_act(float v, int act) {
  switch (act) {
    case TALOS_ACT_RELU: return v > 0.f ? v : 0.f;
    case TALOS_ACT_TANH: return talos_tanh(v);
    case TALOS_ACT_SILU: return v / (1.f + __expf(-v));
    default: return v;
  }
}
// Derivative evaluated on the saved tensor: the OUTPUT for relu/tanh, the PRE-activation for silu.
__device__ __forceinline__ float talos_dact(float s, int act) {
  switch (act) {
    case TALOS_ACT_RELU: return s > 0.f ? 1.f : 0.f;
    case TALOS_ACT_TANH: return 1.f - s * s;
    case TALOS_ACT_SILU: { float g = 1.f / (1.f + __expf(-s)); return g * (1.f + s * (1.f - g)); }
    default: return 1.f;
  }
}

// Epilogue in device form (see talos_epilogue in the public header for the order of operations).
struct EpiArgs {
  const float* bias; float* aux_out; long long ld_aux_out; const float* aux_in; long long ld_aux_in;
  int act; int dact; int beta;
};
inline EpiArgs talos_epi_args(const talos_epilogue* e) {
  EpiArgs a{nullptr, nullptr, 0, nullptr, 0, 0, 0, 0};
  if (e) { a.bias = e->bias; a.aux_out = e->aux_out; a.ld_aux_out = e->ld_aux_out; a.aux_in = e->aux_in;
           a.ld_aux_in = e->ld_aux_in; a.act = e->act; a.dact = e->dact; a.beta = e->beta; }
  return a;
}
__device__ __forceinline__ float talos_epilogue_apply(const EpiArgs& e, float acc, long long m, long long n,
                                                      const float* C, long long ldc) {
  float v = acc;
  if (e.bias) v += e.bias[n];
  if (e.aux_out) e.aux_out[m * e.ld_aux_out + n] = v;
  if (e.act) v = talos_act(v, e.act);
  if (e.aux_in && e.dact) v *= talos_dact(e.aux_in[m * e.ld_aux_in + n], e.dact);
  if (e.beta) v += C[m * ldc + n];
  return v;
}

// Whether a product's result (or the pre-activation it saves) overlaps an operand.  Such a product is sound only while ONE tile
// spans its columns, so that a CTA has read its rows of A before it writes them (y = act(x.W) with y over x, a square layer): it
// keeps the widest tile of its route, and the dispatch rules that would hand it to narrower ones ask here first.
inline bool talos_result_over_operand(int opA, int opB, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, int64_t strideA, const float* B, int64_t ldb,
                                      int64_t strideB, const float* C, int64_t ldc, int64_t strideC, int64_t batch, const EpiArgs& e) {
  if (K == 0) return false;
  auto extent = [&](int64_t rows, int64_t cols, int64_t ld, int64_t stride) { return (rows - 1) * ld + cols + (batch > 1 ? (batch - 1) * stride : 0); };
  const int64_t na = opA == TALOS_OP_N ? extent(M, K, lda, strideA) : extent(K, M, lda, strideA);
  const int64_t nb = opB == TALOS_OP_N ? extent(K, N, ldb, strideB) : extent(N, K, ldb, strideB);
  auto hits = [&](const float* p, int64_t n) { return p && ((A < p + n && p < A + na) || (B < p + n && p < B + nb)); };
  return hits(C, extent(M, N, ldc, strideC)) || hits(e.aux_out, extent(M, N, e.ld_aux_out, 0));
}

// Internal cross-file entry points.
void talos_gemm_fp32_launch(talos_ctx* ctx, int opA, int opB, int64_t M, int64_t N, int64_t K, const float* A,
                            int64_t lda, int64_t strideA, const float* B, int64_t ldb, int64_t strideB, float* C,
                            int64_t ldc, int64_t strideC, int64_t batch, const EpiArgs& epi);
void talos_gemm_small_launch(talos_ctx* ctx, int opA, int opB, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, int64_t strideA, const float* B,
                             int64_t ldb, int64_t strideB, float* C, int64_t ldc, int64_t strideC, int64_t batch, const EpiArgs& epi);
// Reduction elements that one CTA of these kernels walks for a plain product.
int64_t talos_gemm_small_walk(talos_ctx* ctx, int64_t M, int64_t N, int64_t K);
bool talos_linear_bwd_small_launch(talos_ctx* ctx, const float* x, const float* W, const float* saved, const float* dy, float* dx, float* dW, float* db,
                                   int64_t rows, int64_t in_f, int64_t out_f, int act, int accumulate);
// Returns false when the shape/alignment is not eligible (caller falls back to the fp32 kernel).
// First stage of the column sums only: dZ = dY * act'(saved) when dact != 0 (dz may alias dy) and the per-slab column
// sums of dZ left in `partial` ([slabs][n]); returns the slab count, 0 (nothing launched) when the shape is not served.
// The PPO loss kernel without its statistics pass: per-block {loss, kl} sums into partial[blocks][2] (returns blocks =
// ceil(n / 128)) and, when colsum_part is given, per-block column sums of [dlogits | dvalue | 0...] into
// colsum_part[blocks][cs_width] (only where talos_ppo_loss_colsum_supported says so).
int talos_ppo_loss_launch(talos_ctx* ctx, const float* logits, int64_t ld_logits, const float* values, int64_t value_stride, const int32_t* actions,
                          const float* old_logp, const float* adv, const float* ret, int64_t n, int32_t n_actions, float clip, float c_value,
                          float c_entropy, float denom, float* dlogits, int64_t ld_out, float* dvalues, int64_t dvalue_stride, float* partial,
                          float* colsum_part, int cs_width);
bool talos_ppo_loss_colsum_supported(int32_t n_actions, int cs_width);
int talos_colsum_partials_launch(talos_ctx* ctx, const float* dy, float* dz, const float* saved, int dact, int64_t rows, int64_t n,
                                 float* partial, int64_t cap);
// Optional extras for callers that run the same products every step (the PPO trainer):
//  * b_hi / b_lo: the B operand already prepared by the caller with the same shape and pitch as B -- in 3xTF32 mode its
//    TF32 hi / lo split, in TF32 mode b_hi = B rounded to TF32 (b_lo unused) -- so the per-call preparation kernel is
//    skipped (weights change once per optimizer step, not once per product);
//  * partial / partial_floats / splits_out: when the product is split along K, leave the `*splits_out` partial results
//    [splits][M][N] in `partial` (dense, pitch N) and do NOT reduce them into C -- the caller reduces several products'
//    partials in one launch.  *splits_out = 1 means C was written directly (no split, or `partial` too small).
struct TcExtra {
  const float* b_hi = nullptr; const float* b_lo = nullptr;
  float* partial = nullptr; size_t partial_floats = 0; int* splits_out = nullptr;
  // Fused hidden-layer input gradient: C = (A.B^T) * (1 - tanh_saved^2) and per-slab column sums of C into colsum_part
  // ([*colsum_slabs_out][N], summed by the caller).  *colsum_slabs_out stays 0 when the launch did not take the fused
  // route: C is then the plain product and the caller applies the factor itself.
  const float* tanh_saved = nullptr; int64_t ld_saved = 0; float* colsum_part = nullptr; size_t colsum_floats = 0; int* colsum_slabs_out = nullptr;
};
bool talos_gemm_tc_launch(talos_ctx* ctx, int opA, int opB, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda,
                          const float* B, int64_t ldb, float* C, int64_t ldc, int mode, const EpiArgs& epi, const TcExtra* extra = nullptr);
// dZ = dY * act'(saved) (dz may alias dy) and db (+)= column sums of dZ in one pass over the rows; false when the
// shape is not served by the vector kernel (n % 4 != 0, n > 1024 or unaligned), in which case nothing was launched.
bool talos_dact_colsum_launch(talos_ctx* ctx, const float* dy, float* dz, const float* saved, int dact, float* db, int64_t rows, int64_t n,
                              int accumulate);
bool talos_gemm_tc_launch_batched(talos_ctx* ctx, int opA, int opB, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda,
                                  int64_t strideA, const float* B, int64_t ldb, int64_t strideB, float* C, int64_t ldc, int64_t strideC,
                                  int64_t batch, int mode, const EpiArgs& epi);
