// Host-side internal declarations shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/krans_cuda.h"
#include "kr_types.cuh"

#include <cstdlib>

// Cap on the dynamic shared memory a one-block solve uses for its CG vectors
// (KRANS_SMEM_CG_KB, default 0: global memory). Measured on B200: 160 KiB
// gave 8% less CG time on a 1000-unknown solve and cost 16% of a batch of
// uneven solves, whose cluster teams lose L1 capacity to the carve-out. Larger
// carve-outs leave less of the SM's 256 KiB to the L1 cache.
inline size_t cta_smem_cap() {
  static const size_t cap = [] {
    const char *e = getenv("KRANS_SMEM_CG_KB");
    return (size_t)(e ? atoll(e) : 0) * 1024;
  }();
  return cap;
}

namespace kr {

void set_error(const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what, const char *file, int line);

#define KR_CUDA(call)                                                                       \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess)                                                                  \
      return ::kr::cuda_fail(e_, #call, __FILE__, __LINE__);                               \
  } while (0)

#define KR_CHECK_ARG(cond, msg)                                                             \
  do {                                                                                      \
    if (!(cond)) {                                                                          \
      ::kr::set_error("%s", msg);                                                           \
      return KRANS_ERR_INVALID_ARGUMENT;                                                    \
    }                                                                                       \
  } while (0)

struct RngState;
struct GridBarrierState;

} // namespace kr

struct krans_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  size_t budget = 0;
  std::atomic<size_t> in_use{0}; // device bytes allocated through dev_alloc* (the server thread allocates too)
  int sms = 0;
  int cc_major = 0, cc_minor = 0;
  double *h_scalar = nullptr; // pinned scalars for D2H reads
  double *d_scalar = nullptr; // device scalars (reductions)
  double *d_partials = nullptr;
  int partial_blocks = 0;
  krans_batch_tuning tune{16384, 120000, 8, {1, 2, 4, 8, 16, 32}}; // batched-launch knobs in effect
  std::mutex mu;
  // Kept scratch of the calls that work on the context's stream (see ws_take)
  std::mutex ws_mu;
  cudaMemPool_t pool = nullptr; // of the kept scratch and of the second copies of matrices (see kPoolKeep)
  char *ws = nullptr;
  size_t ws_bytes = 0;
  bool ws_busy = false;
  std::mutex copies_mu;
  std::vector<krans_mat *> copied; // matrices with second copies
  // blocks of a single solve's cluster: cyclic FP64, cyclic mixed, LOBPCG (-1: not asked yet; under mu)
  int solo_cluster[3] = {-1, -1, -1};
};

namespace kr {
// An operand cut by columns for the standalone SpMV (kr_spmv.cu): part q holds
// every row's entries in columns [cols q / parts, cols (q + 1) / parts), in
// storage order, as CSR of its own.
constexpr int kMaxParts = 8;
struct SpmvParts {
  int parts = 0; // 0: not cut
  int32_t *rp[kMaxParts] = {};
  int32_t *ci = nullptr;
  double *v64 = nullptr;
  float *v32 = nullptr;
};
// A second copy of a matrix's entries, kept for speed alone: the sorted slices of
// A and A^T that the solvers read, or A^T cut by columns. A matrix does without
// where there is no room, and in a context with a budget, which is for what the
// callers ask for (a planted FP64 matrix takes 20 bytes an entry, and 47 with its
// slices). Where a later allocation finds no room, the copies that nothing uses go
// back to the device. What launches work with a copy holds it (hold_slices, hold_cut),
// from when its own memory is allocated until its kernels are done, or queued on
// the context's stream.
struct SpeedCopy {
  krans_ctx *ctx = nullptr;
  char *base = nullptr;
  size_t bytes = 0;
  SlicedView sl{}, slT{}; // slices = 0: that operand has none
  SpmvParts cut;          // parts = 0: not cut
  std::atomic<bool> captured{false}; // a graph may replay launches that read it: it stays with its matrix
  ~SpeedCopy();           // frees it in the order of the context's stream
};
} // namespace kr

struct krans_mat {
  krans_ctx *ctx = nullptr;
  int64_t m = 0, n = 0, nnz = 0;
  int32_t *rp = nullptr, *ci = nullptr, *rpT = nullptr, *ciT = nullptr;
  double *v = nullptr, *vT = nullptr;
  float *v32 = nullptr, *vT32 = nullptr;
  int lanes = 1, lanesT = 1;
  int32_t ulen = 0, ulenT = 0; // uniform row length of A / A^T (0 = not uniform)
  krans_spmv_tuning tune{}, tuneT{}; // standalone SpMV kernel of A / A^T (zero: automatic)
  // under the context's copies_mu:
  std::shared_ptr<kr::SpeedCopy> slices; // sorted slices of A / A^T for the solvers
  std::shared_ptr<kr::SpeedCopy> cut;    // A^T cut by columns, where its x is larger than L2
  char *base = nullptr;         // one device allocation holding every stored array
  size_t bytes = 0;
};

struct krans_vec {
  krans_ctx *ctx = nullptr;
  int64_t n = 0;
  double *d = nullptr;
};

struct krans_rng {
  krans_ctx *ctx = nullptr;
  kr::RngState *d = nullptr;
  uint32_t seed = 0;
  int mode = 0;
};

namespace kr {
// One stored operand (A or its transpose) as the standalone SpMV sees it.
struct SpmvOperand {
  int64_t rows, cols, nnz;
  const int32_t *rp, *ci;
  const double *v64;
  const float *v32;
  int lanes;
  int32_t ulen;
  krans_spmv_tuning tune;
  const SpmvParts *cut; // or nullptr
};
inline SpmvOperand spmv_operand(const krans_mat *A, int trans, const SpeedCopy *cut) {
  return trans ? SpmvOperand{A->n, A->m, A->nnz, A->rpT, A->ciT, A->vT, A->vT32, A->lanesT, A->ulenT, A->tuneT,
                             cut ? &cut->cut : nullptr}
               : SpmvOperand{A->m, A->n, A->nnz, A->rp, A->ci, A->v, A->v32, A->lanes, A->ulen, A->tune, nullptr};
}
// y = op x on `s` (kr_spmv.cu); fp32: FP32 values and sums
cudaError_t spmv_launch(const SpmvOperand &A, bool fp32, const double *x, double *y, int sms, cudaStream_t s);
int spmv_rows_per_block(int64_t rows, int64_t nnz);
// allocation with budget accounting
bool over_budget(const krans_ctx *ctx, size_t bytes); // these on top of what is allocated
int dev_alloc(krans_ctx *ctx, void **p, size_t bytes);
cudaError_t dev_malloc(krans_ctx *ctx, void **p, size_t bytes); // without the budget
void dev_free(krans_ctx *ctx, void *p, size_t bytes);
// Scratch of one call on the context's stream, kept from call to call: a
// cudaMalloc and cudaFree per call cost 0.3 ms and more (the three block products
// of a 36-column block: 1.35 ms a round with them). One call holds it at a time,
// another (a nested solve, another thread) gets an allocation of its own. What a
// call has queued may still use it after ws_give: the next holder queues on the
// same stream. At most kWsKeep bytes are kept; a call that needs more, or finds
// the device short, allocates for itself, and idle scratch goes back to the
// device before an allocation fails. A context with a budget keeps none: it
// would count against calls that fit beside what the callers themselves hold.
constexpr size_t kWsKeep = (size_t)256 << 20;
// The kept scratch and the second copies come from a pool of the context's own. The
// device's default pool gives freed memory back at the next wait of a stream,
// whoever's: the first product after a matrix of 16.8M rows was destroyed took 48
// ms. This one keeps kPoolKeep unused bytes, gives back what is above when a matrix
// is destroyed, and all of it when the device is full.
constexpr size_t kPoolKeep = (size_t)64 << 20;
struct WsHold {
  void *p = nullptr;
  size_t bytes = 0;
  enum { kNone, kKept, kOwn, kOwnAsync, kOwnUncounted } mode = kNone;
};
// What a call that does not get the kept scratch allocates for itself
enum class WsOwn {
  kDevice,    // cudaMalloc; the caller has waited for its kernels when it gives it back
  kStream,    // freed in stream order (it need not have waited)
  kUncounted, // the same, and the budget does not count it
};
int ws_take(krans_ctx *ctx, size_t bytes, WsHold *w, WsOwn own = WsOwn::kDevice);
void ws_give(krans_ctx *ctx, WsHold *w);
// Stream-ordered forms (cudaMallocAsync / cudaFreeAsync on `s`): neither
// waits for kernels running on other streams, unlike cudaFree, which waits
// for the whole device. The served paths use them so that releasing one
// finished launch never waits for a persistent launch still resident.
int dev_alloc_async(krans_ctx *ctx, void **p, size_t bytes, cudaStream_t s);
// Loads every kernel of the library into the context when it is created.
// With CUDA's lazy module loading (the default), the first launch of a kernel
// loads it, and loading may wait for the kernels already running: a first
// launch beside a resident persistent launch (a new precision or solver in
// the server, a standalone SpMV) would wait until that launch ends. Each
// kernel translation unit lists its kernels in a preload_* function.
void preload(const void *kernel);
void preload_capi_kernels();
void preload_spmv_kernels();
void preload_gram_kernels();
void preload_batch_cta_kernels();
void preload_batch_cluster_kernels();
void preload_cyclic_grid_kernels();
void preload_lobpcg_kernels();
void preload_lobpcg_cta_kernels();
void preload_lobpcg_cluster_kernels();
void dev_free_async(krans_ctx *ctx, void *p, size_t bytes, cudaStream_t s);
int pick_lanes(int64_t rows, int64_t nnz);
// threads per row of the solvers' SpMV from the context's tuning table
inline int tuned_lanes(const krans_ctx *ctx, int64_t rows, int64_t nnz) {
  const double mean = rows > 0 ? (double)nnz / (double)rows : 0.0;
  const double bound[5] = {3.0, 8.0, 16.0, 32.0, 64.0};
  int b = 0;
  while (b < 5 && mean > bound[b])
    b++;
  return ctx->tune.lanes[b];
}
// Team of a single solve by its size m + n (KRANS_TEAM_AUTO): one block below
// the first line, a cluster of 16 blocks between them, the whole GPU from the
// second on. One block costs the least per step and many blocks the least per
// entry. Measured (ms), incidence matrices of mean degree 6, mixed precision, one
// block / cluster / whole GPU: m + n = 4000: 22.8 / 25.4 / 44; 8000: 43 / 27.8 /
// 48; 32000: 162 / 37 / 58; 64000: 377 / 58 / 67; 128000: - / 84 / 68. Block
// LOBPCG: 5000: 98 / 76 / 96; 10000: 174 / 95 / 119; 30000: 390 / 113 / 128; 60000:
// 839 / 155 / 147.
constexpr int64_t kSoloClusterMin = 5000, kSoloGridMin = 100000;
constexpr int64_t kSoloLobpcgClusterMin = 4000, kSoloLobpcgGridMin = 40000;
// While a server lives on the device, a solve stays on one block up to here: the
// server's resident launch leaves few SMs free, which one block finds and a
// cluster or the whole GPU would have to wait for.
constexpr int64_t kServedGridMin = 120000;
// live servers of this process on a device
std::atomic<int> &device_servers(int device);
// the copies as they are now, or nullptr
inline std::shared_ptr<SpeedCopy> hold_slices(const krans_mat *A) {
  std::lock_guard<std::mutex> lk(A->ctx->copies_mu);
  return A->slices;
}
inline std::shared_ptr<SpeedCopy> hold_cut(const krans_mat *A) {
  std::lock_guard<std::mutex> lk(A->ctx->copies_mu);
  return A->cut;
}
// A (or its stored transpose) as the solvers' device code sees it; `slices` as held
inline CsrView csr_view(const krans_mat *A, bool trans, const SpeedCopy *slices) {
  const SlicedView none{};
  if (trans)
    return CsrView{A->n, A->m, A->nnz, A->rpT, A->ciT, A->vT, A->vT32, tuned_lanes(A->ctx, A->n, A->nnz), A->ulenT,
                   slices ? slices->slT : none};
  return CsrView{A->m, A->n, A->nnz, A->rp, A->ci, A->v, A->v32, tuned_lanes(A->ctx, A->m, A->nnz), A->ulen,
                 slices ? slices->sl : none};
}
} // namespace kr
