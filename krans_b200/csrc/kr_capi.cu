// C ABI of the KraNS B200 engine: context, CSR matrices, vectors, SpMV,
// random vectors and the single-request solver launches.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "kr_device.cuh"
#include "kr_internal.h"

namespace kr {

static thread_local std::string g_last_error;

void set_error(const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  g_last_error = buf;
}

int cuda_fail(cudaError_t e, const char *what, const char *file, int line) {
  set_error("CUDA error %s (%s) in %s at %s:%d", cudaGetErrorName(e), cudaGetErrorString(e), what,
            file, line);
  if (e == cudaErrorMemoryAllocation)
    return KRANS_ERR_OUT_OF_MEMORY;
  return KRANS_ERR_CUDA;
}

static void release_bytes(krans_ctx *ctx, size_t bytes) {
  size_t cur = ctx->in_use.load();
  while (!ctx->in_use.compare_exchange_weak(cur, cur - std::min(cur, bytes))) {
  }
}

bool over_budget(const krans_ctx *ctx, size_t bytes) {
  return ctx->budget && ctx->in_use.load() + bytes > ctx->budget;
}
static int budget_fail(krans_ctx *ctx, size_t bytes) {
  set_error("HBM budget exceeded: %zu + %zu > %zu bytes", ctx->in_use.load(), bytes, ctx->budget);
  return KRANS_ERR_OUT_OF_MEMORY;
}

static bool give_back(krans_ctx *ctx);
// Both forms of a device allocation: once more if the context had something to
// give back. An error is the caller's to report: the next launch's check must
// not find it.
cudaError_t dev_malloc(krans_ctx *ctx, void **p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation && give_back(ctx))
    e = cudaMalloc(p, bytes);
  if (e != cudaSuccess)
    cudaGetLastError();
  return e;
}
static cudaError_t stream_malloc(krans_ctx *ctx, void **p, size_t bytes, cudaStream_t s) {
  cudaError_t e = cudaMallocAsync(p, bytes, s);
  if (e == cudaErrorMemoryAllocation && give_back(ctx))
    e = cudaMallocAsync(p, bytes, s);
  if (e != cudaSuccess)
    cudaGetLastError();
  return e;
}
int dev_alloc(krans_ctx *ctx, void **p, size_t bytes) {
  *p = nullptr;
  if (bytes == 0)
    bytes = 256;
  if (over_budget(ctx, bytes))
    return budget_fail(ctx, bytes);
  const cudaError_t e = dev_malloc(ctx, p, bytes);
  if (e != cudaSuccess)
    return cuda_fail(e, "cudaMalloc", __FILE__, __LINE__);
  ctx->in_use.fetch_add(bytes);
  return KRANS_OK;
}

// Frees the kept scratch in stream order (cudaFree would wait for the whole
// device, a server's resident launch included). Call with ws_mu held.
static void ws_drop(krans_ctx *ctx) {
  if (!ctx->ws)
    return;
  cudaFreeAsync(ctx->ws, ctx->stream);
  release_bytes(ctx, ctx->ws_bytes);
  ctx->ws = nullptr;
  ctx->ws_bytes = 0;
}

static bool ws_release(krans_ctx *ctx) { // true if there was idle scratch
  std::lock_guard<std::mutex> lk(ctx->ws_mu);
  if (!ctx->ws || ctx->ws_busy)
    return false;
  ws_drop(ctx);
  return true;
}

static uint64_t pool_bytes(krans_ctx *ctx, cudaMemPoolAttr what) {
  uint64_t v = 0;
  if (!ctx->pool || cudaMemPoolGetAttribute(ctx->pool, what, &v) != cudaSuccess)
    return 0;
  return v;
}

// When the device has no room: what the context holds beyond its callers' own
// allocations goes back, from the context's pool to the device. False if there
// was nothing.
static bool give_back(krans_ctx *ctx) {
  cudaGetLastError(); // the failed allocation's
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)
    return false;
  bool any = ws_release(ctx);
  {
    std::lock_guard<std::mutex> lk(ctx->copies_mu);
    for (krans_mat *A : ctx->copied)
      for (auto *c : {&A->slices, &A->cut})
        if (*c && c->use_count() == 1 && !(*c)->captured) { // nothing but the matrix holds it
          c->reset();
          any = true;
        }
  }
  if (!any && pool_bytes(ctx, cudaMemPoolAttrReservedMemCurrent) <= pool_bytes(ctx, cudaMemPoolAttrUsedMemCurrent))
    return false;
  cudaStreamSynchronize(ctx->stream);
  cudaMemPoolTrimTo(ctx->pool, 0);
  return true;
}

SpeedCopy::~SpeedCopy() {
  cudaFreeAsync(base, ctx->stream);
  release_bytes(ctx, bytes);
}
// Room for a second copy, or nullptr
static std::shared_ptr<SpeedCopy> copy_alloc(krans_ctx *ctx, size_t bytes) {
  char *p = nullptr;
  if (ctx->budget)
    return nullptr;
  if (cudaMallocFromPoolAsync((void **)&p, bytes, ctx->pool, ctx->stream) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  ctx->in_use.fetch_add(bytes);
  auto c = std::make_shared<SpeedCopy>();
  c->ctx = ctx;
  c->base = p;
  c->bytes = bytes;
  return c;
}

int ws_take(krans_ctx *ctx, size_t bytes, WsHold *w, WsOwn own) {
  *w = WsHold{};
  if (!ctx->budget && bytes <= kWsKeep) {
    std::lock_guard<std::mutex> lk(ctx->ws_mu);
    if (!ctx->ws_busy) {
      if (ctx->ws_bytes < bytes) {
        // grown by half again, so that a run of growing calls reallocates a few times only
        const size_t want = std::min(kWsKeep, std::max(bytes + bytes / 2, (size_t)1 << 20));
        ws_drop(ctx);
        if (cudaMallocFromPoolAsync((void **)&ctx->ws, want, ctx->pool, ctx->stream) == cudaSuccess) {
          ctx->ws_bytes = want;
          ctx->in_use.fetch_add(want);
        } else {
          cudaGetLastError();
          ctx->ws = nullptr;
        }
      }
      if (ctx->ws) {
        ctx->ws_busy = true;
        w->p = ctx->ws;
        w->bytes = bytes;
        w->mode = WsHold::kKept;
        return KRANS_OK;
      }
    }
  }
  if (own == WsOwn::kUncounted) {
    KR_CUDA(stream_malloc(ctx, &w->p, bytes, ctx->stream));
    w->mode = WsHold::kOwnUncounted;
    return KRANS_OK;
  }
  const bool async = own == WsOwn::kStream;
  const int rc = async ? dev_alloc_async(ctx, &w->p, bytes, ctx->stream) : dev_alloc(ctx, &w->p, bytes);
  if (rc == KRANS_OK) {
    w->bytes = bytes;
    w->mode = async ? WsHold::kOwnAsync : WsHold::kOwn;
  }
  return rc;
}

void ws_give(krans_ctx *ctx, WsHold *w) {
  if (w->mode == WsHold::kKept) {
    std::lock_guard<std::mutex> lk(ctx->ws_mu);
    ctx->ws_busy = false;
  } else if (w->mode == WsHold::kOwn) {
    dev_free(ctx, w->p, w->bytes);
  } else if (w->mode == WsHold::kOwnAsync) {
    dev_free_async(ctx, w->p, w->bytes, ctx->stream);
  } else if (w->mode == WsHold::kOwnUncounted) {
    cudaFreeAsync(w->p, ctx->stream);
  }
  *w = WsHold{};
}

void dev_free(krans_ctx *ctx, void *p, size_t bytes) {
  if (!p)
    return;
  if (bytes == 0)
    bytes = 256;
  cudaFree(p);
  release_bytes(ctx, bytes);
}

int dev_alloc_async(krans_ctx *ctx, void **p, size_t bytes, cudaStream_t s) {
  *p = nullptr;
  if (bytes == 0)
    bytes = 256;
  if (over_budget(ctx, bytes))
    return budget_fail(ctx, bytes);
  const cudaError_t e = stream_malloc(ctx, p, bytes, s);
  if (e != cudaSuccess)
    return cuda_fail(e, "cudaMallocAsync", __FILE__, __LINE__);
  ctx->in_use.fetch_add(bytes);
  return KRANS_OK;
}

void dev_free_async(krans_ctx *ctx, void *p, size_t bytes, cudaStream_t s) {
  if (!p)
    return;
  if (bytes == 0)
    bytes = 256;
  cudaFreeAsync(p, s);
  release_bytes(ctx, bytes);
}

// Threads per row of the SpMV. Short rows go one per thread: the gathers of
// these operators are random sectors, and a thread walking a short row keeps
// the most of them in flight per instruction (measured on B200: the F^T of a
// shift operator, 2 entries per row, runs 1.5x faster with 1 lane than with 2;
// an incidence matrix's F^T, 6 entries per row on average, is fastest with 2).
int pick_lanes(int64_t rows, int64_t nnz) {
  const double mean = rows > 0 ? (double)nnz / (double)rows : 0.0;
  if (mean <= 3.0)
    return 1;
  if (mean <= 8.0)
    return 2;
  if (mean <= 16.0)
    return 4;
  if (mean <= 32.0)
    return 8;
  if (mean <= 64.0)
    return 16;
  return 32;
}

// Deterministic dot product in one launch: a partial per block, and the block
// that finishes last sums them in index order. `out` may be pinned host memory,
// so that a scalar the host waits for takes one launch and no copy (a caller's own
// Golub-Kahan step of 1000 unknowns, seven scalars among its twelve calls: 157 us
// with two launches and a copy each, 127 us so).
__global__ void __launch_bounds__(256) dot_kernel(int64_t n, const double *x, const double *y, double *part,
                                                  unsigned *done, double *out, int take_sqrt) {
  __shared__ TeamShared sh;
  __shared__ bool s_last;
  int buf = 0;
  double v[1] = {0.0};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    v[0] += x[i] * y[i];
  block_sum<1>(&sh, buf, v);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v[0];
    __threadfence();
    s_last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last)
    return;
  __threadfence();
  v[0] = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x)
    v[0] += __ldcg(part + i);
  block_sum<1>(&sh, buf, v);
  if (threadIdx.x == 0) {
    out[0] = take_sqrt ? sqrt(v[0]) : v[0];
    *done = 0; // for the next launch on the stream
  }
}
// the same in two launches without a counter, for krans_vec_dot_noalloc: partial per block, then one block sums
__global__ void __launch_bounds__(256) dot_partial_kernel(int64_t n, const double *x, const double *y,
                                                          double *part) {
  __shared__ TeamShared sh;
  int buf = 0;
  double v[1] = {0.0};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    v[0] += x[i] * y[i];
  block_sum<1>(&sh, buf, v);
  if (threadIdx.x == 0)
    part[blockIdx.x] = v[0];
}
__global__ void __launch_bounds__(256) sum_partials_kernel(int nb, const double *part, double *out,
                                                           int take_sqrt) {
  __shared__ TeamShared sh;
  int buf = 0;
  double v[1] = {0.0};
  for (int i = threadIdx.x; i < nb; i += blockDim.x)
    v[0] += part[i];
  block_sum<1>(&sh, buf, v);
  if (threadIdx.x == 0)
    out[0] = take_sqrt ? sqrt(v[0]) : v[0];
}
__global__ void axpy_kernel(int64_t n, double a, const double *x, double *y) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] += a * x[i];
}
__global__ void scale_kernel(int64_t n, double a, double *x) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] *= a;
}
__global__ void scale_by_inv_norm_kernel(int64_t n, const double *nrm, double *x) {
  const double s = nrm[0];
  if (!(s > 0.0))
    return;
  const double a = 1.0 / s;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] *= a;
}
__global__ void fill_kernel(int64_t n, double a, double *x) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = a;
}
__global__ void to_f32_kernel(int64_t n, const double *x, float *y) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = (float)x[i];
}

// ---- deterministic transpose: count, scan, scatter, per-row sort, gather ----
__global__ void col_count_kernel(int64_t nnz, const int32_t *ci, int32_t *cnt) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(cnt + ci[k], 1);
}
// exclusive scan of cnt[0..n) into out[0..n]; single block, 8 consecutive values
// per thread and round: sums by warp shuffles, two barriers a round (1024 values
// and 22 barriers a round: the device's part of creating a 200003-column incidence
// matrix took 402 us, and takes 251)
__global__ void __launch_bounds__(1024) scan_kernel(int64_t n, const int32_t *cnt, int32_t *out) {
  constexpr int V = 8;
  __shared__ int32_t s_warp[2][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int32_t carry = 0;
  int buf = 0;
  for (int64_t base = 0; base < n; base += 1024 * V, buf ^= 1) {
    const int64_t i0 = base + (int64_t)threadIdx.x * V;
    int32_t v[V], sum = 0;
#pragma unroll
    for (int k = 0; k < V; k++) {
      v[k] = i0 + k < n ? cnt[i0 + k] : 0;
      sum += v[k];
    }
    int32_t run = sum; // inclusive over the warp
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(0xffffffffu, run, o);
      run += lane >= o ? t : 0;
    }
    if (lane == 31)
      s_warp[buf][wid] = run;
    __syncthreads();
    const int32_t w = s_warp[buf][lane];
    const int32_t before = __reduce_add_sync(0xffffffffu, lane < wid ? w : 0);
    const int32_t total = __reduce_add_sync(0xffffffffu, w);
    int32_t at = carry + before + run - sum;
#pragma unroll
    for (int k = 0; k < V; k++) {
      if (i0 + k < n)
        out[i0 + k] = at;
      at += v[k];
    }
    carry += total; // the next round writes the other buffer
  }
  if (threadIdx.x == 0)
    out[n] = carry;
}
__global__ void scatter_kernel(int64_t nnz, const int32_t *ci, int32_t *cursor, int32_t *perm) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += (int64_t)gridDim.x * blockDim.x) {
    const int32_t pos = atomicAdd(cursor + ci[k], 1);
    perm[pos] = (int32_t)k;
  }
}
// sort each transposed row's source positions ascending (warp per row):
// rows up to 32 entries in registers (bitonic), longer rows by ranking.
__global__ void row_sort_kernel(int64_t rows, const int32_t *rp, int32_t *perm, int32_t *tmp) {
  const int lane = threadIdx.x & 31;
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = w; r < rows; r += nw) {
    const int32_t b = rp[r], e = rp[r + 1], L = e - b;
    if (L <= 1)
      continue;
    if (L <= 32) {
      int32_t v = lane < L ? perm[b + lane] : INT32_MAX;
      for (int k = 2; k <= 32; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
          const int32_t o = __shfl_xor_sync(0xffffffffu, v, j);
          const bool up = ((lane & k) == 0);
          const bool lower = ((lane & j) == 0);
          v = (lower == up) ? min(v, o) : max(v, o);
        }
      if (lane < L)
        perm[b + lane] = v;
    } else {
      for (int32_t i = lane; i < L; i += 32) {
        const int32_t key = perm[b + i];
        int32_t rank = 0;
        for (int32_t j = 0; j < L; j++)
          rank += perm[b + j] < key;
        tmp[b + rank] = key;
      }
      __syncwarp();
      for (int32_t i = lane; i < L; i += 32)
        perm[b + i] = tmp[b + i];
    }
  }
}
__global__ void row_of_kernel(int64_t m, const int32_t *rp, int32_t *rowof) {
  const int lane = threadIdx.x & 31;
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = w; r < m; r += nw)
    for (int32_t k = rp[r] + lane; k < rp[r + 1]; k += 32)
      rowof[k] = (int32_t)r;
}
__global__ void gather_t_kernel(int64_t nnz, const int32_t *perm, const int32_t *rowof, const double *v,
                                int32_t *ciT, double *vT) {
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += (int64_t)gridDim.x * blockDim.x) {
    const int32_t k = perm[p];
    ciT[p] = rowof[k];
    vT[p] = v[k];
  }
}

// Sorted slices of a CSR operand (SlicedView): one block per window of
// kSliceWindow rows ranks them by length, longest first (ties by row, so the
// order is deterministic), and writes the slots' rows and the slices' widths.
__global__ void __launch_bounds__(kSliceWindow) slice_sort_kernel(int64_t rows, const int32_t *rp, int32_t *row,
                                                                  int32_t *width) {
  __shared__ int32_t len[kSliceWindow];
  const int t = threadIdx.x;
  const int64_t w0 = (int64_t)blockIdx.x * kSliceWindow, i = w0 + t;
  const int here = (int)imin64(kSliceWindow, rows - w0);
  const int32_t mine = t < here ? rp[i + 1] - rp[i] : -1;
  len[t] = mine;
  __syncthreads();
  int rank = 0;
  for (int j = 0; j < kSliceWindow; j++)
    rank += len[j] > mine || (len[j] == mine && j < t);
  if (w0 + (rank & ~31) < rows) { // the last window's slices past the last row do not exist
    row[w0 + rank] = t < here ? (int32_t)i : -1;
    if ((rank & 31) == 0)
      width[(w0 + rank) >> 5] = mine;
  }
}
// the rounds of every slice, a warp per slice
__global__ void slice_fill_kernel(int64_t slices, const int32_t *off, const int32_t *row, const int32_t *rp,
                                  const int32_t *ci, const double *v, int32_t *sci, double *sv, float *sv32) {
  const int lane = threadIdx.x & 31;
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t s = w; s < slices; s += nw) {
    const int32_t r = row[s * 32 + lane];
    const int32_t b = r >= 0 ? rp[r] : 0, len = r >= 0 ? rp[r + 1] - b : 0;
    const int32_t o0 = off[s], o1 = off[s + 1];
    for (int32_t j = 0; j < o1 - o0; j++) {
      const size_t k = (size_t)(o0 + j) * 32 + lane;
      const double x = j < len ? v[b + j] : 0.0;
      sci[k] = j < len ? ci[b + j] : 0;
      sv[k] = x;
      if (sv32)
        sv32[k] = (float)x;
    }
  }
}

// first entry of row [b, e) in column c or beyond (columns ascending)
KR_DEV int32_t first_from(const int32_t *ci, int32_t b, int32_t e, int64_t c) {
  while (b < e) {
    const int32_t m = b + (e - b) / 2;
    if (ci[m] < c)
      b = m + 1;
    else
      e = m;
  }
  return b;
}
// entries of every row in column part [c0, c1)
__global__ void part_count_kernel(int64_t rows, const int32_t *rp, const int32_t *ci, int64_t c0, int64_t c1,
                                  int32_t *cnt) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t b = first_from(ci, rp[r], rp[r + 1], c0);
    cnt[r] = first_from(ci, b, rp[r + 1], c1) - b;
  }
}
// the part's entries, where its row pointers say (they count the entries of the earlier parts too)
__global__ void part_fill_kernel(int64_t rows, const int32_t *rp, const int32_t *ci, const double *v, int64_t c0,
                                 const int32_t *prp, int32_t *pci, double *pv, float *pv32) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t b = first_from(ci, rp[r], rp[r + 1], c0), k0 = prp[r], len = prp[r + 1] - k0;
    for (int32_t j = 0; j < len; j++) {
      pci[k0 + j] = ci[b + j];
      pv[k0 + j] = v[b + j];
      if (pv32)
        pv32[k0 + j] = (float)v[b + j];
    }
  }
}
__global__ void part_shift_kernel(int64_t n, const int32_t *by, int32_t *rp) { // rp[0..n) += *by
  const int32_t d = *by;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    rp[i] += d;
}

__global__ void __launch_bounds__(1024) rng_mt_kernel(RngState *st, double *out, int64_t n) {
  __shared__ uint32_t ring[6 * 624]; // 936 attempts a round
  block_mt_normals(st, out, n, ring, 6);
}
// Long draws of the same sequence in three steps. One block runs the MT19937
// recurrence alone and stores `states` states (the current one first); all SMs
// then try the polar attempts in them and count the accepted ones per block, and
// again, each block knowing the counts before it, write their normals; one block
// takes over the new state. One block doing all of it spends most of its time in
// log and square root on one SM's FP64 pipe. What is left is the serial
// recurrence, one barrier per state: 24 vectors of 262144 take 5.4 ms (31 ms
// with one block, one state and five barriers a round).
constexpr int kMtTry = 256; // attempts per block
__global__ void __launch_bounds__(640) rng_mt_states_kernel(const RngState *st, uint32_t *words, int64_t states,
                                                            int64_t *last) {
  __shared__ uint32_t ring[2][640]; // a word per thread; the last 16 are not used
  const int i = threadIdx.x, at = min(i, 623);
  if (i == 0)
    *last = -1;
  uint32_t v = st->mt[at];
  ring[0][i] = v;
  if (i < 624)
    words[i] = v;
  __syncthreads();
  for (int64_t b = 1; b < states; b++) {
    v = mt_next_word(ring[(b - 1) & 1], at);
    ring[b & 1][i] = v;
    __syncthreads();
    if (i < 624)
      words[b * 624 + i] = v;
  }
}
__global__ void __launch_bounds__(kMtTry) rng_mt_count_kernel(const RngState *st, const uint32_t *words,
                                                              int64_t states, int32_t *cnt) {
  const int64_t t = (int64_t)blockIdx.x * kMtTry + threadIdx.x, w = st->idx + 4 * t;
  double x, y, r2;
  const int got = __syncthreads_count(w + 3 < states * 624 && polar_attempt(words + w, x, y, r2));
  if (threadIdx.x == 0)
    cnt[blockIdx.x] = got;
}
__global__ void __launch_bounds__(kMtTry) rng_mt_emit_kernel(const RngState *st, const uint32_t *words,
                                                             int64_t states, const int32_t *cnt, double *out,
                                                             int64_t n, int64_t *last, double *saved) {
  __shared__ int s_warp[kMtTry / 32];
  __shared__ int64_t s_before;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t first = st->has_saved ? 1 : 0; // out[0] is the carried value
  const int64_t need = (n - first + 1) >> 1;   // pairs
  // accepted attempts in the blocks before this one
  int64_t sum = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += kMtTry)
    sum += cnt[b];
  for (int o = 16; o > 0; o >>= 1)
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (threadIdx.x == 0)
    s_before = 0;
  __syncthreads();
  if (lane == 0)
    atomicAdd((unsigned long long *)&s_before, (unsigned long long)sum);
  const int64_t t = (int64_t)blockIdx.x * kMtTry + threadIdx.x, w = st->idx + 4 * t;
  double x = 0.0, y = 0.0, r2 = 0.0;
  const bool acc = w + 3 < states * 624 && polar_attempt(words + w, x, y, r2);
  const unsigned bal = __ballot_sync(0xffffffffu, acc);
  if (lane == 0)
    s_warp[wid] = __popc(bal);
  __syncthreads();
  int64_t before = s_before + __popc(bal & ((1u << lane) - 1u));
  for (int v = 0; v < wid; v++)
    before += s_warp[v];
  if (t == 0 && first && n > 0)
    out[0] = st->saved;
  if (acc && before < need) {
    const double mult = polar_scale(r2);
    const int64_t p = first + 2 * before;
    out[p] = __dmul_rn(y, mult);
    if (p + 1 < n)
      out[p + 1] = __dmul_rn(x, mult);
    if (before == need - 1) { // the draw ends here
      *last = w + 3;
      saved[0] = __dmul_rn(x, mult);
    }
  }
}
__global__ void __launch_bounds__(1024) rng_mt_finish_kernel(RngState *st, const uint32_t *words, int64_t states,
                                                             const int32_t *cnt, int blocks, double *out, int64_t n,
                                                             const int64_t *last, const double *saved) {
  __shared__ uint32_t ring[6 * 624];
  __shared__ int64_t s_got;
  const int64_t first = st->has_saved ? 1 : 0, end = *last;
  if (threadIdx.x == 0)
    s_got = 0;
  __syncthreads();
  if (end < 0) { // the states ran out before the draw ended (their number allows for that in one of 1e9 draws)
    int64_t sum = 0;
    for (int b = threadIdx.x; b < blocks; b += blockDim.x)
      sum += cnt[b];
    atomicAdd((unsigned long long *)&s_got, (unsigned long long)sum);
  }
  __syncthreads();
  const int64_t b = end < 0 ? states - 1 : end / 624;
  for (int i = threadIdx.x; i < 624; i += blockDim.x)
    st->mt[i] = words[b * 624 + i];
  const bool odd = ((n - first) & 1) != 0; // the last pair's second value is carried over
  if (threadIdx.x == 0) {
    st->idx = end < 0 ? 624 : (int32_t)(end + 1 - b * 624);
    st->has_saved = end >= 0 && odd;
    if (end >= 0 && odd)
      st->saved = saved[0];
  }
  __threadfence_block();
  __syncthreads();
  if (end < 0) {
    const int64_t pos = first + 2 * s_got;
    block_mt_normals(st, out + pos, n - pos, ring, 6);
  }
}
__global__ void rng_philox_kernel(RngState *st, double *out, int64_t n) {
  const uint64_t key = st->philox_key, base = st->philox_ctr;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = philox_normal(key, base + (uint64_t)i);
}
__global__ void rng_philox_advance(RngState *st, int64_t n) { st->philox_ctr += (uint64_t)n; }

void preload(const void *kernel) {
  cudaFuncAttributes a;
  if (cudaFuncGetAttributes(&a, kernel) != cudaSuccess)
    cudaGetLastError();
}

void preload_capi_kernels() {
  const void *ks[] = {(const void *)dot_kernel,         (const void *)dot_partial_kernel,
                      (const void *)sum_partials_kernel,
                      (const void *)axpy_kernel,        (const void *)scale_kernel,
                      (const void *)scale_by_inv_norm_kernel, (const void *)fill_kernel,
                      (const void *)to_f32_kernel,      (const void *)col_count_kernel,
                      (const void *)scan_kernel,        (const void *)scatter_kernel,
                      (const void *)row_sort_kernel,    (const void *)row_of_kernel,
                      (const void *)gather_t_kernel,    (const void *)slice_sort_kernel,
                      (const void *)slice_fill_kernel,  (const void *)part_count_kernel,
                      (const void *)part_fill_kernel,   (const void *)part_shift_kernel,
                      (const void *)rng_mt_kernel,
                      (const void *)rng_mt_states_kernel, (const void *)rng_mt_count_kernel,
                      (const void *)rng_mt_emit_kernel, (const void *)rng_mt_finish_kernel,
                      (const void *)rng_philox_kernel,  (const void *)rng_philox_advance};
  for (const void *k : ks)
    preload(k);
}

// Whether an operand of `rows` rows keeps sorted slices, and how many entries
// these hold, padding included (0: none). longest: of its rows; ulen: their
// length if they are all equal, else 0; len(i): length of row i. An upper bound
// within twice the entries may stand for the number.
// Rows of one entry gain nothing (one load in flight per lane: 5400 of them on one
// block 12.6 us a product, 9.6 with vector loads and four rows in flight), and rows
// of exactly 2 are read with vector loads as they are; rows of fewer than 2 on
// average still gain (the transpose of a shift operator: a CG iteration at 4000
// columns 12.8 -> 10.9 us, at 100000 36 -> 29 us). Padding is read by every product
// and takes memory: at most 7 entries for each real one (one row of 64 among 256
// rows of one makes 6: 11.6 us a product on the whole GPU, 25 with lanes).
template <class Len>
static int64_t slice_entries(int64_t rows, int64_t nnz, int32_t longest, int32_t ulen, Len len) {
  if (nnz == 0 || longest < 2 || longest > kSliceMaxLen || ulen == 2)
    return 0;
  if (ulen)
    return (rows + 31) / 32 * 32 * ulen;
  // Every slice of a window but the first is no wider than the shortest row before
  // it, so the padding of a window is at most 32 times its longest row. Where that is
  // close enough it is taken: counting lengths costs 1 ns a row (a creation with 200003
  // columns takes 3.6 ms).
  int64_t most = nnz;
  for (int64_t w0 = 0; w0 < rows; w0 += kSliceWindow) {
    const int64_t w1 = std::min<int64_t>(rows, w0 + kSliceWindow);
    int32_t top = 0;
    for (int64_t i = w0; i < w1; i++)
      top = std::max(top, len(i));
    most += 32 * (int64_t)top;
  }
  if (most <= 2 * nnz)
    return most;
  // a slice is as wide as the row it starts at, in the order of slice_sort_kernel
  int64_t e = 0;
  for (int64_t w0 = 0; w0 < rows; w0 += kSliceWindow) {
    int32_t of_len[2][kSliceMaxLen + 1] = {}; // two counters a length: rows in turn, shorter chains
    const int64_t w1 = std::min<int64_t>(rows, w0 + kSliceWindow);
    for (int64_t i = w0; i < w1; i++)
      of_len[i & 1][len(i)]++;
    int32_t before = 0; // longer rows
    for (int32_t l = longest; l > 0; l--) {
      const int32_t after = before + of_len[0][l] + of_len[1][l];
      e += 32 * (int64_t)l * ((after + 31) / 32 - (before + 31) / 32);
      before = after;
    }
  }
  return e <= 8 * nnz ? e : 0;
}

static int grid_for(krans_ctx *ctx, int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)ctx->sms * 8;
  if (b > cap)
    b = cap;
  if (b < 1)
    b = 1;
  return (int)b;
}

} // namespace kr

using namespace kr;

extern "C" {

const char *krans_last_error(void) { return kr::g_last_error.c_str(); }
const char *krans_version(void) { return "krans_b200 0.1 (sm_100a)"; }

int krans_abi_sizes(int64_t *out, int capacity) {
  const int64_t sz[9] = {(int64_t)sizeof(krans_cyclic_opts),    (int64_t)sizeof(krans_cyclic_result),
                         (int64_t)sizeof(krans_lobpcg_opts),    (int64_t)sizeof(krans_lobpcg_result),
                         (int64_t)sizeof(krans_request),        (int64_t)sizeof(krans_request_result),
                         (int64_t)sizeof(krans_server_opts),    (int64_t)sizeof(krans_spmv_tuning),
                         (int64_t)sizeof(krans_batch_tuning)};
  for (int i = 0; i < 9 && i < capacity && out; i++)
    out[i] = sz[i];
  return 9;
}

int krans_ctx_create(int device, size_t hbm_budget_bytes, krans_ctx **out) {
  KR_CHECK_ARG(out, "krans_ctx_create: out is NULL");
  *out = nullptr;
  int ndev = 0;
  KR_CUDA(cudaGetDeviceCount(&ndev));
  KR_CHECK_ARG(device >= 0 && device < ndev, "krans_ctx_create: no such device");
  KR_CUDA(cudaSetDevice(device));
  auto *c = new krans_ctx();
  c->device = device;
  c->budget = hbm_budget_bytes;
  cudaDeviceProp prop;
  cudaError_t e = cudaGetDeviceProperties(&prop, device);
  if (e != cudaSuccess) {
    delete c;
    return cuda_fail(e, "cudaGetDeviceProperties", __FILE__, __LINE__);
  }
  c->sms = prop.multiProcessorCount;
  c->cc_major = prop.major;
  c->cc_minor = prop.minor;
  if (prop.major != 10) {
    delete c;
    set_error("krans_ctx_create: device %d is sm_%d%d; this library targets sm_100a (B200)", device,
              prop.major, prop.minor);
    return KRANS_ERR_RUNTIME;
  }
  e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    e = cudaMemPoolCreate(&c->pool, &props);
  }
  if (e == cudaSuccess) {
    uint64_t never = ~0ull; // given back by hand
    e = cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &never);
  }
  if (e == cudaSuccess)
    e = cudaMallocHost(&c->h_scalar, 64 * sizeof(double));
  c->partial_blocks = c->sms * 8;
  if (e == cudaSuccess)
    e = cudaMalloc(&c->d_scalar, 64 * sizeof(double));
  if (e == cudaSuccess)
    e = cudaMalloc(&c->d_partials, (size_t)c->partial_blocks * sizeof(double));
  if (e == cudaSuccess)
    e = cudaMemsetAsync(c->d_scalar, 0, 64 * sizeof(double), c->stream); // scalars, and the block counter of dot_kernel
  if (e != cudaSuccess) {
    int rc = cuda_fail(e, "context setup", __FILE__, __LINE__);
    krans_ctx_destroy(c);
    return rc;
  }
  preload_capi_kernels();
  preload_spmv_kernels();
  preload_gram_kernels();
  preload_batch_cta_kernels();
  preload_batch_cluster_kernels();
  preload_cyclic_grid_kernels();
  preload_lobpcg_kernels();
  preload_lobpcg_cta_kernels();
  preload_lobpcg_cluster_kernels();
  *out = c;
  return KRANS_OK;
}

int krans_ctx_destroy(krans_ctx *ctx) {
  if (!ctx)
    return KRANS_OK;
  cudaSetDevice(ctx->device);
  if (ctx->stream)
    cudaStreamSynchronize(ctx->stream);
  ws_release(ctx);
  if (ctx->h_scalar)
    cudaFreeHost(ctx->h_scalar);
  if (ctx->d_scalar)
    cudaFree(ctx->d_scalar);
  if (ctx->d_partials)
    cudaFree(ctx->d_partials);
  if (ctx->stream)
    cudaStreamSynchronize(ctx->stream); // the scratch is free
  if (ctx->pool)
    cudaMemPoolDestroy(ctx->pool);
  if (ctx->stream)
    cudaStreamDestroy(ctx->stream);
  delete ctx;
  return KRANS_OK;
}

int krans_ctx_synchronize(krans_ctx *ctx) {
  KR_CHECK_ARG(ctx, "NULL context");
  KR_CUDA(cudaStreamSynchronize(ctx->stream));
  return KRANS_OK;
}

int krans_ctx_memory_in_use(const krans_ctx *ctx, size_t *bytes) {
  KR_CHECK_ARG(ctx && bytes, "NULL argument");
  *bytes = ctx->in_use.load(); // kept scratch included
  return KRANS_OK;
}

int krans_ctx_sm_count(const krans_ctx *ctx, int *sms) {
  KR_CHECK_ARG(ctx && sms, "NULL argument");
  *sms = ctx->sms;
  return KRANS_OK;
}

int krans_ctx_set_batch_tuning(krans_ctx *ctx, const krans_batch_tuning *t) {
  KR_CHECK_ARG(ctx && t, "krans_ctx_set_batch_tuning: NULL argument");
  KR_CHECK_ARG(t->cluster_min >= 0 && t->pair_max >= 0, "krans_ctx_set_batch_tuning: negative size threshold");
  KR_CHECK_ARG(t->cluster_size == 0 || (t->cluster_size >= 2 && t->cluster_size <= 16),
               "krans_ctx_set_batch_tuning: cluster_size must be 0 or 2..16");
  for (int b = 0; b < 6; b++)
    KR_CHECK_ARG(t->lanes[b] == 0 || (t->lanes[b] >= 1 && t->lanes[b] <= 32 && (t->lanes[b] & (t->lanes[b] - 1)) == 0),
                 "krans_ctx_set_batch_tuning: lanes must be 0 or a power of two up to 32");
  const krans_batch_tuning def{16384, 120000, 8, {1, 2, 4, 8, 16, 32}};
  std::lock_guard<std::mutex> lk(ctx->mu);
  krans_batch_tuning &u = ctx->tune;
  u.cluster_min = t->cluster_min ? t->cluster_min : def.cluster_min;
  u.pair_max = t->pair_max ? t->pair_max : def.pair_max;
  u.cluster_size = t->cluster_size ? t->cluster_size : def.cluster_size;
  for (int b = 0; b < 6; b++)
    u.lanes[b] = t->lanes[b] ? t->lanes[b] : def.lanes[b];
  return KRANS_OK;
}

int krans_ctx_get_batch_tuning(const krans_ctx *ctx, krans_batch_tuning *t) {
  KR_CHECK_ARG(ctx && t, "krans_ctx_get_batch_tuning: NULL argument");
  *t = ctx->tune;
  return KRANS_OK;
}

int krans_ctx_stream(const krans_ctx *ctx, void **stream) {
  KR_CHECK_ARG(ctx && stream, "NULL argument");
  *stream = (void *)ctx->stream;
  return KRANS_OK;
}

// ---------------------------------------------------------------------------
// CSR
// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// Self-test of the bounded grid barrier: block 0 waits at a barrier that
// block 1 never reaches (it returns at once), so the wait must run out after
// the state's timeout and leave KRANS_ERR_TIMEOUT in the status word.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(64) barrier_timeout_probe_kernel(GridBarrierState *gb, int *status,
                                                                   double *gpart) {
  __shared__ TeamShared sh;
  if (blockIdx.x != 0)
    return;
  TeamGrid tm{&sh, status, gb, gpart, 0, 0};
  tm.sync();
}

extern "C" int krans_selftest_barrier_timeout(krans_ctx *ctx, double timeout_ms, int *status_out,
                                              double *elapsed_ms) {
  KR_CHECK_ARG(ctx && status_out, "krans_selftest_barrier_timeout: NULL argument");
  KR_CHECK_ARG(timeout_ms > 0.0 && timeout_ms <= 10000.0,
               "krans_selftest_barrier_timeout: timeout_ms must be in (0, 10000]");
  KR_CUDA(cudaSetDevice(ctx->device));
  std::lock_guard<std::mutex> lk(ctx->mu);
  struct Probe {
    GridBarrierState gb;
    int status;
    int pad;
    double gpart[2 * 2 * KR_MDOT];
  };
  Probe *d = nullptr;
  int rc = dev_alloc(ctx, (void **)&d, sizeof(Probe));
  if (rc != KRANS_OK)
    return rc;
  Probe h;
  memset(&h, 0, sizeof h);
  h.gb.timeout_ns = (uint64_t)(timeout_ms * 1e6);
  cudaStream_t s = ctx->stream;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t e = cudaMemcpyAsync(d, &h, sizeof h, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaEventCreate(&e0);
  if (e == cudaSuccess)
    e = cudaEventCreate(&e1);
  if (e == cudaSuccess)
    e = cudaEventRecord(e0, s);
  if (e == cudaSuccess) {
    GridBarrierState *gb = &d->gb;
    int *st = &d->status;
    double *gp = d->gpart;
    void *args[] = {(void *)&gb, (void *)&st, (void *)&gp};
    e = cudaLaunchCooperativeKernel((const void *)barrier_timeout_probe_kernel, dim3(2), dim3(64), args, 0, s);
  }
  if (e == cudaSuccess)
    e = cudaEventRecord(e1, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&h, d, sizeof h, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(s);
  float ms = 0.f;
  if (e == cudaSuccess)
    e = cudaEventElapsedTime(&ms, e0, e1);
  if (e0)
    cudaEventDestroy(e0);
  if (e1)
    cudaEventDestroy(e1);
  dev_free(ctx, d, sizeof(Probe));
  if (e != cudaSuccess)
    return cuda_fail(e, "krans_selftest_barrier_timeout", __FILE__, __LINE__);
  *status_out = h.status;
  if (elapsed_ms)
    *elapsed_ms = ms;
  return KRANS_OK;
}

// Columns from which x outgrows what L2 keeps of it beside the streamed operand
// (gathers a second from x of 34 / 67 / 134 MB: 170 / 146 / 84 billion), and the
// columns a part's piece of x should have at most.
static constexpr int64_t kCutCols = 12582912, kPartCols = 6291456;

// A^T cut into column parts (SpmvParts), queued on the context's stream.
static void cut_transpose(krans_ctx *ctx, krans_mat *A, int32_t *cnt) {
  SpmvParts P;
  const int64_t rows = A->n, cols = A->m, nnz = A->nnz;
  P.parts = (int)std::min<int64_t>(kMaxParts, (cols + kPartCols - 1) / kPartCols);
  // fewer than an entry a row and part: y would cost more than x; parts as wide as
  // kCutCols: their pieces of x outgrow L2 too
  if (cols < kCutCols || cols >= P.parts * kCutCols || nnz < rows * P.parts)
    return;
  Carver lay;
  auto carve = [&](Carver &c) {
    for (int q = 0; q < P.parts; q++)
      P.rp[q] = c.take<int32_t>(rows + 1);
    P.ci = c.take<int32_t>(nnz);
    P.v64 = c.take<double>(nnz);
    P.v32 = A->vT32 ? c.take<float>(nnz) : nullptr;
  };
  carve(lay);
  auto copy = copy_alloc(ctx, lay.off + 256);
  if (!copy)
    return;
  Carver c;
  c.base = copy->base;
  carve(c);
  cudaStream_t s = ctx->stream;
  const int g = grid_for(ctx, rows);
  for (int q = 0; q < P.parts; q++) {
    const int64_t c0 = cols * q / P.parts, c1 = cols * (q + 1) / P.parts;
    part_count_kernel<<<g, 256, 0, s>>>(rows, A->rpT, A->ciT, c0, c1, cnt);
    scan_kernel<<<1, 1024, 0, s>>>(rows, cnt, P.rp[q]);
    if (q > 0) // after the entries of the parts before it
      part_shift_kernel<<<g, 256, 0, s>>>(rows + 1, P.rp[q - 1] + rows, P.rp[q]);
    part_fill_kernel<<<g, 256, 0, s>>>(rows, A->rpT, A->ciT, A->vT, c0, P.rp[q], P.ci, P.v64, P.v32);
  }
  copy->cut = P;
  A->cut = std::move(copy);
}

int krans_csr_create(krans_ctx *ctx, int64_t m, int64_t n, int64_t nnz, const int32_t *row_ptr,
                     const int32_t *col_idx, const double *values, int flags, krans_mat **out) {
  KR_CHECK_ARG(ctx && out, "krans_csr_create: NULL argument");
  *out = nullptr;
  KR_CHECK_ARG(m >= 0 && n >= 0 && nnz >= 0, "krans_csr_create: negative size");
  KR_CHECK_ARG(m < INT32_MAX && n < INT32_MAX && nnz < INT32_MAX,
               "krans_csr_create: sizes must fit 32-bit indices");
  KR_CHECK_ARG(row_ptr && (nnz == 0 || (col_idx && values)), "krans_csr_create: NULL array");
  KR_CHECK_ARG(row_ptr[0] == 0 && row_ptr[m] == nnz, "krans_csr_create: row_ptr[0] != 0 or row_ptr[m] != nnz");
  // one pass over the rows (monotone, uniform length) and one over the
  // columns (range, per-column counts for the transpose's uniform length)
  const int64_t L = m > 0 ? (int64_t)(row_ptr[1] - row_ptr[0]) : 0;
  bool uni = m > 0 && L > 0 && L <= 8;
  int32_t longest = 0, longestT = 0;
  for (int64_t i = 0; i < m; i++) {
    const int32_t len = row_ptr[i + 1] - row_ptr[i];
    KR_CHECK_ARG(len >= 0, "krans_csr_create: row_ptr not monotone");
    uni = uni && len == L;
    longest = std::max(longest, len);
  }
  std::vector<int32_t> cc((size_t)n, 0);
  for (int64_t k = 0; k < nnz; k++) {
    const int32_t c = col_idx[k];
    KR_CHECK_ARG(c >= 0 && c < n, "krans_csr_create: column index out of range");
    cc[(size_t)c]++;
  }
  const int32_t LT = n > 0 ? cc[0] : 0;
  bool uniT = n > 0 && LT > 0 && LT <= 8;
  for (int64_t j = 0; j < n; j++) {
    uniT = uniT && cc[(size_t)j] == LT;
    longestT = std::max(longestT, cc[(size_t)j]);
  }
  if (!(flags & (KRANS_CSR_FP64 | KRANS_CSR_FP32)))
    flags |= KRANS_CSR_FP64;
  flags |= KRANS_CSR_FP64; // FP64 values are kept for every path (polish, residuals)
  KR_CUDA(cudaSetDevice(ctx->device));
  const bool f32 = (flags & KRANS_CSR_FP32) != 0;
  const size_t sz_rp = (size_t)(m + 1) * 4, sz_rpT = (size_t)(n + 1) * 4, sz_ci = (size_t)std::max<int64_t>(nnz, 1) * 4;
  const size_t sz_v = (size_t)std::max<int64_t>(nnz, 1) * 8, sz_v32 = (size_t)std::max<int64_t>(nnz, 1) * 4;
  // the stored arrays share one allocation (carved at 256-byte offsets)
  auto up = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const int64_t sl = slice_entries(m, nnz, longest, uni ? (int32_t)L : 0,
                                   [&](int64_t i) { return row_ptr[i + 1] - row_ptr[i]; });
  const int64_t slT = slice_entries(n, nnz, longestT, uniT ? LT : 0, [&](int64_t j) { return cc[(size_t)j]; });
  const size_t total = up(sz_rp) + 2 * up(sz_ci) + 2 * up(sz_v) + up(sz_rpT) + (f32 ? 2 * up(sz_v32) : 0);
  char *base = nullptr;
  int rc = dev_alloc(ctx, (void **)&base, total);
  if (rc != KRANS_OK)
    return rc;
  auto *A = new krans_mat();
  A->ctx = ctx;
  A->m = m;
  A->n = n;
  A->nnz = nnz;
  A->base = base;
  A->bytes = total;
  size_t off = 0;
  auto take = [&](size_t b) {
    char *p = base + off;
    off += up(b);
    return p;
  };
  A->rp = (int32_t *)take(sz_rp);
  A->ci = (int32_t *)take(sz_ci);
  A->v = (double *)take(sz_v);
  A->rpT = (int32_t *)take(sz_rpT);
  A->ciT = (int32_t *)take(sz_ci);
  A->vT = (double *)take(sz_v);
  if (f32) {
    A->v32 = (float *)take(sz_v32);
    A->vT32 = (float *)take(sz_v32);
  }
  // the slices of both operands, in an allocation of their own
  auto carve_slices = [&](Carver &c, int64_t rows, int64_t e, int32_t longest_row) {
    const int64_t nsl = (rows + 31) / 32;
    SlicedView S;
    S.slices = (int32_t)nsl;
    S.longest = longest_row;
    S.row = c.take<int32_t>(nsl * 32);
    S.off = c.take<int32_t>(nsl + 1);
    S.ci = c.take<int32_t>(e);
    S.v64 = c.take<double>(e);
    S.v32 = f32 ? c.take<float>(e) : nullptr;
    return S;
  };
  if (sl || slT) {
    SlicedView S{}, ST{};
    auto carve = [&](Carver &c) {
      if (sl)
        S = carve_slices(c, m, sl, longest);
      if (slT)
        ST = carve_slices(c, n, slT, longestT);
    };
    Carver lay;
    carve(lay);
    if ((A->slices = copy_alloc(ctx, lay.off + 256))) {
      Carver c;
      c.base = A->slices->base;
      carve(c);
      A->slices->sl = S;
      A->slices->slT = ST;
    }
  }
  // scratch of the device transpose: kept by the context and used in stream
  // order, so releasing it does not wait for the device, and the next matrix's
  // host work overlaps this matrix's transpose kernels
  cudaStream_t s = ctx->stream;
  WsHold scr;
  const size_t sz_w = up((size_t)(std::max(m, n) / 32 + 1) * 4); // slice widths, one operand at a time
  const size_t sz_scr = up(sz_rpT) + 3 * up(sz_ci) + sz_w;
  rc = ws_take(ctx, sz_scr, &scr, WsOwn::kUncounted); // gone when this returns: the budget is for what stays
  if (rc != KRANS_OK) {
    krans_csr_destroy(A);
    return rc;
  }
  cudaError_t e = cudaSuccess;
  int32_t *scratch = (int32_t *)scr.p;
  int32_t *cnt = scratch, *perm = (int32_t *)((char *)scratch + up(sz_rpT));
  int32_t *tmp = (int32_t *)((char *)perm + up(sz_ci)), *rowof = (int32_t *)((char *)tmp + up(sz_ci));
  int32_t *width = (int32_t *)((char *)rowof + up(sz_ci));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(A->rp, row_ptr, sz_rp, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && nnz)
    e = cudaMemcpyAsync(A->ci, col_idx, (size_t)nnz * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && nnz)
    e = cudaMemcpyAsync(A->v, values, (size_t)nnz * 8, cudaMemcpyHostToDevice, s);
  // the host arrays may be reused once this returns: wait for the copies only
  cudaEvent_t copied = nullptr;
  if (e == cudaSuccess)
    e = cudaEventCreateWithFlags(&copied, cudaEventDisableTiming);
  if (e == cudaSuccess)
    e = cudaEventRecord(copied, s);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(cnt, 0, sz_rpT, s);
  if (e == cudaSuccess && nnz) {
    const int g = grid_for(ctx, nnz);
    col_count_kernel<<<g, 256, 0, s>>>(nnz, A->ci, cnt);
    scan_kernel<<<1, 1024, 0, s>>>(n, cnt, A->rpT);
    e = cudaMemcpyAsync(cnt, A->rpT, (size_t)n * 4, cudaMemcpyDeviceToDevice, s);
    scatter_kernel<<<g, 256, 0, s>>>(nnz, A->ci, cnt, perm);
    row_sort_kernel<<<grid_for(ctx, n * 32), 256, 0, s>>>(n, A->rpT, perm, tmp);
    row_of_kernel<<<grid_for(ctx, m * 32), 256, 0, s>>>(m, A->rp, rowof);
    gather_t_kernel<<<g, 256, 0, s>>>(nnz, perm, rowof, A->v, A->ciT, A->vT);
    if (f32) {
      to_f32_kernel<<<g, 256, 0, s>>>(nnz, A->v, A->v32);
      to_f32_kernel<<<g, 256, 0, s>>>(nnz, A->vT, A->vT32);
    }
    auto fill = [&](int64_t rows, const int32_t *rp, const int32_t *ci, const double *v, const SlicedView &S) {
      int32_t *off = const_cast<int32_t *>(S.off), *row = const_cast<int32_t *>(S.row);
      slice_sort_kernel<<<(unsigned)((rows + kSliceWindow - 1) / kSliceWindow), kSliceWindow, 0, s>>>(rows, rp, row, width);
      scan_kernel<<<1, 1024, 0, s>>>(S.slices, width, off);
      slice_fill_kernel<<<grid_for(ctx, (int64_t)S.slices * 32), 256, 0, s>>>(
          S.slices, off, row, rp, ci, v, const_cast<int32_t *>(S.ci), const_cast<double *>(S.v64),
          const_cast<float *>(S.v32));
    };
    if (A->slices && sl)
      fill(m, A->rp, A->ci, A->v, A->slices->sl);
    if (A->slices && slT)
      fill(n, A->rpT, A->ciT, A->vT, A->slices->slT);
    cut_transpose(ctx, A, cnt);
  } else if (e == cudaSuccess) {
    e = cudaMemsetAsync(A->rpT, 0, sz_rpT, s);
  }
  if (e == cudaSuccess)
    e = cudaGetLastError();
  if (copied) {
    const cudaError_t es = cudaEventSynchronize(copied);
    if (e == cudaSuccess)
      e = es;
    cudaEventDestroy(copied);
  }
  ws_give(ctx, &scr); // the kernels queued above use it in stream order
  if (e != cudaSuccess) {
    cudaStreamSynchronize(s);
    rc = cuda_fail(e, "krans_csr_create", __FILE__, __LINE__);
    krans_csr_destroy(A);
    return rc;
  }
  A->lanes = pick_lanes(m, nnz);
  A->lanesT = pick_lanes(n, nnz);
  // uniform row lengths (e.g. incidence and difference operators) let the
  // SpMV skip the row pointers and use vector loads
  A->ulen = uni ? (int32_t)L : 0;
  A->ulenT = uniT ? LT : 0;
  if (A->slices || A->cut) {
    std::lock_guard<std::mutex> lk(ctx->copies_mu);
    ctx->copied.push_back(A);
  }
  *out = A;
  return KRANS_OK;
}

int krans_csr_destroy(krans_mat *A) {
  if (!A)
    return KRANS_OK;
  {
    std::lock_guard<std::mutex> lk(A->ctx->copies_mu);
    auto &all = A->ctx->copied;
    all.erase(std::remove(all.begin(), all.end(), A), all.end());
  }
  krans_ctx *ctx = A->ctx;
  const bool copies = A->slices || A->cut;
  A->slices.reset();
  A->cut.reset();
  dev_free(ctx, A->base, A->bytes); // waits for the device
  if (copies && cudaStreamSynchronize(ctx->stream) == cudaSuccess) // which tells the pool that the copies are free
    cudaMemPoolTrimTo(ctx->pool, (size_t)pool_bytes(ctx, cudaMemPoolAttrUsedMemCurrent) + kPoolKeep);
  delete A;
  return KRANS_OK;
}

int krans_csr_dims(const krans_mat *A, int64_t *m, int64_t *n, int64_t *nnz) {
  KR_CHECK_ARG(A, "NULL matrix");
  if (m)
    *m = A->m;
  if (n)
    *n = A->n;
  if (nnz)
    *nnz = A->nnz;
  return KRANS_OK;
}

int krans_csr_device_arrays(const krans_mat *A, int trans, const int32_t **row_ptr,
                            const int32_t **col_idx, const double **values, const float **values32) {
  KR_CHECK_ARG(A, "NULL matrix");
  if (row_ptr)
    *row_ptr = trans ? A->rpT : A->rp;
  if (col_idx)
    *col_idx = trans ? A->ciT : A->ci;
  if (values)
    *values = trans ? A->vT : A->v;
  if (values32)
    *values32 = trans ? A->vT32 : A->v32;
  return KRANS_OK;
}

// ---------------------------------------------------------------------------
// vectors
// ---------------------------------------------------------------------------
int krans_vec_create(krans_ctx *ctx, int64_t n, krans_vec **out) {
  KR_CHECK_ARG(ctx && out, "krans_vec_create: NULL argument");
  KR_CHECK_ARG(n >= 0, "krans_vec_create: negative size");
  *out = nullptr;
  auto *v = new krans_vec();
  v->ctx = ctx;
  v->n = n;
  int rc = dev_alloc(ctx, (void **)&v->d, (size_t)std::max<int64_t>(n, 1) * 8);
  if (rc != KRANS_OK) {
    delete v;
    return rc;
  }
  cudaError_t e = cudaMemsetAsync(v->d, 0, (size_t)std::max<int64_t>(n, 1) * 8, ctx->stream);
  if (e != cudaSuccess) {
    dev_free(ctx, v->d, (size_t)std::max<int64_t>(n, 1) * 8);
    delete v;
    return cuda_fail(e, "cudaMemsetAsync", __FILE__, __LINE__);
  }
  *out = v;
  return KRANS_OK;
}

int krans_vec_destroy(krans_vec *v) {
  if (!v)
    return KRANS_OK;
  dev_free(v->ctx, v->d, (size_t)std::max<int64_t>(v->n, 1) * 8);
  delete v;
  return KRANS_OK;
}

int krans_vec_size(const krans_vec *v, int64_t *n) {
  KR_CHECK_ARG(v && n, "NULL argument");
  *n = v->n;
  return KRANS_OK;
}

int krans_vec_device_ptr(krans_vec *v, double **dptr) {
  KR_CHECK_ARG(v && dptr, "NULL argument");
  *dptr = v->d;
  return KRANS_OK;
}

int krans_vec_upload(krans_vec *v, const double *host, int64_t n) {
  KR_CHECK_ARG(v && (host || n == 0), "NULL argument");
  KR_CHECK_ARG(n == v->n, "krans_vec_upload: size mismatch");
  if (n)
    KR_CUDA(cudaMemcpyAsync(v->d, host, (size_t)n * 8, cudaMemcpyHostToDevice, v->ctx->stream));
  KR_CUDA(cudaStreamSynchronize(v->ctx->stream));
  return KRANS_OK;
}

int krans_vec_download(const krans_vec *v, double *host, int64_t n) {
  KR_CHECK_ARG(v && (host || n == 0), "NULL argument");
  KR_CHECK_ARG(n == v->n, "krans_vec_download: size mismatch");
  if (n)
    KR_CUDA(cudaMemcpyAsync(host, v->d, (size_t)n * 8, cudaMemcpyDeviceToHost, v->ctx->stream));
  KR_CUDA(cudaStreamSynchronize(v->ctx->stream));
  return KRANS_OK;
}

static void launch_dot(krans_ctx *c, int64_t n, const double *x, const double *y, int take_sqrt, double *out) {
  const int g = std::min<int>(grid_for(c, n), c->partial_blocks);
  dot_kernel<<<g, 256, 0, c->stream>>>(n, x, y, c->d_partials, reinterpret_cast<unsigned *>(c->d_scalar + 1), out,
                                       take_sqrt);
}
static int reduce_to_host(krans_ctx *c, int64_t n, const double *x, const double *y, int take_sqrt,
                          double *out) {
  launch_dot(c, n, x, y, take_sqrt, c->h_scalar); // pinned: the device writes it directly
  KR_CUDA(cudaGetLastError());
  KR_CUDA(cudaStreamSynchronize(c->stream));
  *out = *(volatile double *)c->h_scalar;
  return KRANS_OK;
}

int krans_vec_dot(const krans_vec *x, const krans_vec *y, double *out) {
  KR_CHECK_ARG(x && y && out, "NULL argument");
  KR_CHECK_ARG(x->n == y->n, "krans_vec_dot: size mismatch");
  return reduce_to_host(x->ctx, x->n, x->d, y->d, 0, out);
}

int krans_vec_nrm2(const krans_vec *v, double *out) {
  KR_CHECK_ARG(v && out, "NULL argument");
  return reduce_to_host(v->ctx, v->n, v->d, v->d, 1, out);
}

int krans_vec_axpy(krans_vec *y, double alpha, const krans_vec *x) {
  KR_CHECK_ARG(x && y, "NULL argument");
  KR_CHECK_ARG(x->n == y->n, "krans_vec_axpy: size mismatch");
  axpy_kernel<<<grid_for(y->ctx, y->n), 256, 0, y->ctx->stream>>>(y->n, alpha, x->d, y->d);
  KR_CUDA(cudaGetLastError());
  return KRANS_OK;
}

int krans_vec_scale(krans_vec *v, double alpha) {
  KR_CHECK_ARG(v, "NULL argument");
  scale_kernel<<<grid_for(v->ctx, v->n), 256, 0, v->ctx->stream>>>(v->n, alpha, v->d);
  KR_CUDA(cudaGetLastError());
  return KRANS_OK;
}

int krans_vec_normalize(krans_vec *v) {
  KR_CHECK_ARG(v, "NULL argument");
  krans_ctx *c = v->ctx;
  launch_dot(c, v->n, v->d, v->d, 1, c->d_scalar);
  scale_by_inv_norm_kernel<<<grid_for(c, v->n), 256, 0, c->stream>>>(v->n, c->d_scalar, v->d);
  KR_CUDA(cudaGetLastError());
  return KRANS_OK;
}

int krans_vec_fill(krans_vec *v, double value) {
  KR_CHECK_ARG(v, "NULL argument");
  fill_kernel<<<grid_for(v->ctx, v->n), 256, 0, v->ctx->stream>>>(v->n, value, v->d);
  KR_CUDA(cudaGetLastError());
  return KRANS_OK;
}

int krans_vec_copy(krans_vec *dst, const krans_vec *src) {
  KR_CHECK_ARG(dst && src, "NULL argument");
  KR_CHECK_ARG(dst->n == src->n, "krans_vec_copy: size mismatch");
  if (dst->n)
    KR_CUDA(cudaMemcpyAsync(dst->d, src->d, (size_t)dst->n * 8, cudaMemcpyDeviceToDevice, dst->ctx->stream));
  return KRANS_OK;
}

int krans_vec_clone(const krans_vec *src, krans_vec **out) {
  KR_CHECK_ARG(src && out, "NULL argument");
  int rc = krans_vec_create(src->ctx, src->n, out);
  if (rc != KRANS_OK)
    return rc;
  return krans_vec_copy(*out, src);
}

int krans_spmv_ex(const krans_mat *A, int trans, int precision, const krans_vec *x, krans_vec *y) {
  KR_CHECK_ARG(A && x && y, "krans_spmv: NULL argument");
  const int64_t rows = trans ? A->n : A->m, cols = trans ? A->m : A->n;
  KR_CHECK_ARG(x->n == cols && y->n == rows, "krans_spmv: size mismatch");
  KR_CHECK_ARG(precision == KRANS_PREC_FP64 || precision == KRANS_PREC_MIXED, "krans_spmv: unknown precision");
  KR_CHECK_ARG(precision != KRANS_PREC_MIXED || A->v32,
               "krans_spmv: matrix has no FP32 values (create with KRANS_CSR_FP32)");
  krans_ctx *c = A->ctx;
  const auto cut = trans ? hold_cut(A) : nullptr;
  if (cut && !cut->captured) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    KR_CUDA(cudaStreamIsCapturing(c->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone)
      cut->captured = true;
  }
  KR_CUDA(spmv_launch(spmv_operand(A, trans, cut.get()), precision == KRANS_PREC_MIXED, x->d, y->d, c->sms, c->stream));
  return KRANS_OK;
}

int krans_csr_set_spmv_tuning(krans_mat *A, int trans, const krans_spmv_tuning *t) {
  KR_CHECK_ARG(A && t, "krans_csr_set_spmv_tuning: NULL argument");
  KR_CHECK_ARG(t->kernel >= KRANS_SPMV_AUTO && t->kernel <= KRANS_SPMV_LANES,
               "krans_csr_set_spmv_tuning: unknown kernel");
  KR_CHECK_ARG(t->rows_per_block >= 0 && t->rows_per_block <= 2048,
               "krans_csr_set_spmv_tuning: rows_per_block outside 0..2048");
  KR_CHECK_ARG(t->x_evict_last == 0 || t->x_evict_last == 1, "krans_csr_set_spmv_tuning: x_evict_last must be 0 or 1");
  const int32_t ulen = trans ? A->ulenT : A->ulen;
  KR_CHECK_ARG(t->kernel != KRANS_SPMV_UNIFORM || ulen == 1 || ulen == 2 || ulen == 4,
               "krans_csr_set_spmv_tuning: UNIFORM needs every row to hold exactly 1, 2 or 4 entries");
  (trans ? A->tuneT : A->tune) = *t;
  return KRANS_OK;
}

int krans_csr_get_spmv_tuning(const krans_mat *A, int trans, krans_spmv_tuning *t) {
  KR_CHECK_ARG(A && t, "krans_csr_get_spmv_tuning: NULL argument");
  *t = trans ? A->tuneT : A->tune;
  return KRANS_OK;
}

int krans_spmv(const krans_mat *A, int trans, const krans_vec *x, krans_vec *y) {
  return krans_spmv_ex(A, trans, KRANS_PREC_FP64, x, y);
}

// ---------------------------------------------------------------------------
// RNG
// ---------------------------------------------------------------------------
static void mt_seed_host(RngState &s, uint32_t seed) {
  s.mt[0] = seed;
  for (int i = 1; i < 624; i++)
    s.mt[i] = 1812433253u * (s.mt[i - 1] ^ (s.mt[i - 1] >> 30)) + (uint32_t)i;
  s.idx = 624;
  s.has_saved = 0;
  s.saved = 0.0;
}

int krans_rng_create(krans_ctx *ctx, uint32_t seed, int mode, krans_rng **out) {
  KR_CHECK_ARG(ctx && out, "krans_rng_create: NULL argument");
  KR_CHECK_ARG(mode == KRANS_RNG_MT19937 || mode == KRANS_RNG_PHILOX, "krans_rng_create: bad mode");
  *out = nullptr;
  if (seed == 0)
    seed = std::random_device{}();
  RngState h;
  memset(&h, 0, sizeof h);
  mt_seed_host(h, seed);
  h.philox_key = ((uint64_t)seed << 32) ^ 0x9E3779B97F4A7C15ull;
  h.philox_ctr = 0;
  h.mode = mode;
  auto *r = new krans_rng();
  r->ctx = ctx;
  r->seed = seed;
  r->mode = mode;
  int rc = dev_alloc(ctx, (void **)&r->d, sizeof(RngState));
  if (rc != KRANS_OK) {
    delete r;
    return rc;
  }
  cudaError_t e = cudaMemcpyAsync(r->d, &h, sizeof h, cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) {
    krans_rng_destroy(r);
    return cuda_fail(e, "rng upload", __FILE__, __LINE__);
  }
  *out = r;
  return KRANS_OK;
}

int krans_rng_destroy(krans_rng *r) {
  if (!r)
    return KRANS_OK;
  dev_free(r->ctx, r->d, sizeof(RngState));
  delete r;
  return KRANS_OK;
}

int krans_rng_seed(const krans_rng *r, uint32_t *seed) {
  KR_CHECK_ARG(r && seed, "NULL argument");
  *seed = r->seed;
  return KRANS_OK;
}

// Draws from here on run on all SMs; below, one block's single launch is quicker.
static constexpr int64_t kMtLong = 8192, kMtPiece = (int64_t)1 << 22;
int krans_rng_normal(krans_rng *r, krans_vec *out) {
  KR_CHECK_ARG(r && out, "krans_rng_normal: NULL argument");
  krans_ctx *c = r->ctx;
  if (r->mode == KRANS_RNG_PHILOX) {
    rng_philox_kernel<<<grid_for(c, out->n), 256, 0, c->stream>>>(r->d, out->d, out->n);
    rng_philox_advance<<<1, 1, 0, c->stream>>>(r->d, out->n);
  } else {
    // one block draws what is short, what finds no room for scratch, and what is
    // being captured (scratch taken during a capture would belong to the graph)
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    KR_CUDA(cudaStreamIsCapturing(c->stream, &cap));
    const bool one = cap != cudaStreamCaptureStatusNone;
    // Pieces, so that the words stay within the kept scratch. A rest shorter than
    // kMtLong is one block's too: a piece has pairs to draw, also where it starts
    // with a carried value (one of a single value would need none).
    int64_t at = 0;
    for (; !one && out->n - at >= kMtLong; at += std::min(kMtPiece, out->n - at)) {
      const int64_t n = std::min(kMtPiece, out->n - at);
      // attempts for n / 2 accepted ones: mean n / 2 / p and six standard
      // deviations, p = pi / 4; four words each, after the current state
      const double need = 0.5 * (double)(n + 1), p = 0.78539816339744831;
      const int64_t tries = (int64_t)(need / p + 6.0 * std::sqrt(need * (1.0 - p)) / p) + 8;
      const int64_t states = (4 * tries + 623) / 624 + 1;
      const int blocks = (int)((states * 156 + kMtTry - 1) / kMtTry);
      Carver lay;
      lay.take<uint32_t>(states * 624);
      lay.take<int32_t>(blocks);
      lay.take<int64_t>(2);
      WsHold ws;
      if (ws_take(c, lay.off + 256, &ws, WsOwn::kStream) != KRANS_OK) {
        set_error("%s", "");
        cudaGetLastError();
        break;
      }
      Carver cv;
      cv.base = (char *)ws.p;
      uint32_t *words = cv.take<uint32_t>(states * 624);
      int32_t *cnt = cv.take<int32_t>(blocks);
      int64_t *last = cv.take<int64_t>(2);
      double *saved = reinterpret_cast<double *>(last + 1);
      rng_mt_states_kernel<<<1, 640, 0, c->stream>>>(r->d, words, states, last);
      rng_mt_count_kernel<<<blocks, kMtTry, 0, c->stream>>>(r->d, words, states, cnt);
      rng_mt_emit_kernel<<<blocks, kMtTry, 0, c->stream>>>(r->d, words, states, cnt, out->d + at, n, last, saved);
      rng_mt_finish_kernel<<<1, 1024, 0, c->stream>>>(r->d, words, states, cnt, blocks, out->d + at, n, last, saved);
      ws_give(c, &ws);
    }
    if (at < out->n)
      rng_mt_kernel<<<1, 1024, 0, c->stream>>>(r->d, out->d + at, out->n - at);
  }
  KR_CUDA(cudaGetLastError());
  return KRANS_OK;
}

int krans_cyclic_opts_init(krans_cyclic_opts *o) {
  KR_CHECK_ARG(o, "NULL argument");
  memset(o, 0, sizeof *o);
  o->k = 1;
  o->ncv = 48;
  o->max_restarts = 80;
  o->tol_abs = 1e-12;
  o->tol_rel = 1e-10;
  o->reorth = 2;
  o->use_harmonic = 1;
  o->target_tau = 0.0;
  o->nullity_known = -1;
  o->rank_known = -1;
  o->cg_maxit = 80;
  o->cg_rel_tol = 1e-10;
  o->cg_breakdown_tol = 1e-30;
  o->projector_passes = 1;
  o->grad_max_iters = 3000;
  o->frob_samples = 4;
  o->prescreen_factor = 0.8;
  o->stagnation_restarts = 30;
  o->return_left_space = 0;
  o->verbose = 0;
  o->precision = KRANS_PREC_FP64;
  o->team = KRANS_TEAM_AUTO;
  o->precond_aat = KRANS_PRECOND_NONE;
  o->precond_steps = 8;
  o->polish_block = 0;
  o->mixed_fallback = 1;
  return KRANS_OK;
}

int krans_lobpcg_opts_init(krans_lobpcg_opts *o) {
  KR_CHECK_ARG(o, "NULL argument");
  memset(o, 0, sizeof *o);
  o->nev = 1;
  o->block_size = 0;
  o->max_iters = 1000;
  o->tol_abs = 1e-12;
  o->tol_rel = 1e-10;
  o->soft_locking = 1;
  o->restart = 0.9;
  o->gs_tol = 1e-14;
  o->gs_reorth = 1;
  o->frob_samples = 4;
  o->max_tiny_dim = 0;
  o->nullity_known = -1;
  o->rank_known = -1;
  o->progress_every = 100;
  o->precision = KRANS_PREC_FP64;
  o->team = KRANS_TEAM_AUTO;
  o->precond_normal = KRANS_PRECOND_NONE;
  o->precond_steps = 6;
  return KRANS_OK;
}

} // extern "C"
