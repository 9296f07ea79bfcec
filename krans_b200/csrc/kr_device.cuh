// Device building blocks of the KraNS B200 engine.
//
// The solvers are written once against a "team": the set of threads that
// cooperates on one null-space solve.
//   TeamCta  - one thread block (batched serving: many solves side by side,
//              one per block, synchronised with __syncthreads).
//   TeamGrid - every block of a cooperative launch (one large solve on the
//              whole GPU, synchronised with a bounded grid barrier).
//   TeamCluster - the blocks of a thread-block cluster (solves in between).
// All reductions use a fixed tree whose shape depends only on the team size,
// and a batch picks its teams by m + n alone, so a request gives bit-identical
// results in any batch. A single solve picks its own team: other rounding.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/krans_cuda.h"
#include "kr_types.cuh"

#define KR_DEV __device__ __forceinline__
#define KR_MAX_WARPS 32
#define KR_MAX_CLUSTER 16 // blocks of a cluster team
#ifndef KR_RED_K
#define KR_RED_K 8 // values per fused team reduction
#endif
#ifndef KR_SLICE_J
#define KR_SLICE_J 4 // rounds of a slice that team_spmv_sliced keeps in flight
#endif
#ifndef KR_SPMV_ROWS
#define KR_SPMV_ROWS 4 // row groups each warp keeps in flight in team_spmv
#endif

namespace kr {

// ---------------------------------------------------------------------------
// timing / barrier primitives
// ---------------------------------------------------------------------------
KR_DEV uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A grid barrier wait gives up after this long and flags KRANS_ERR_TIMEOUT
// (the longest legitimate wait is a serial section on the leader block).
constexpr uint64_t kBarrierTimeoutNs = 8ull * 1000ull * 1000ull * 1000ull;

#define KR_RED_LD (KR_MAX_WARPS + 2) // row of warp partials: 8 rows of double pairs on distinct banks

// Per-block shared memory used by the team primitives.
struct TeamShared {
  alignas(16) double red[2][KR_RED_K * KR_RED_LD]; // double-buffered warp partials, one row per value
  alignas(16) double dots[KR_MDOT * KR_RED_LD];    // warp partials of team_multidot
  double bc[2][KR_RED_K];                          // broadcast slots (grid reductions)
  double h[160];                                   // Gram-Schmidt coefficients
  double cpart[2][KR_MAX_CLUSTER][KR_MDOT];        // cluster reductions: every block's partials
  int ibuf[64];                                    // small integer scratch
};

KR_DEV double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Warp totals of K values (K = 2, 4 or 8) by recursive halving: at each of the
// first log2 K steps a lane keeps half of the values and gives the other half
// away, then the butterfly goes on with one value. K + 5 - log2 K exchanges
// instead of 5 K, and the same additions in the same tree as K butterflies (a
// lane adds its partner's partial of the same value at offsets 16, 8, 4, 2, 1),
// so the totals are the same to the last bit. Lane l returns the total of
// value l / (32 / K).
template <int K> KR_DEV double warp_sums(double (&v)[K]) {
  static_assert(K == 2 || K == 4 || K == 8, "power of two");
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int half = K / 2; half > 0; half /= 2, o /= 2) {
    const bool hi = lane & o;
#pragma unroll
    for (int k = 0; k < half; k++) {
      const double keep = hi ? v[k + half] : v[k], give = hi ? v[k] : v[k + half];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  double t = v[0];
  for (; o > 0; o /= 2)
    t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// sum of a row of warp partials in warp order
KR_DEV double sum_warps(const double *r, int nw) {
  double s = 0.0;
  int w = 0;
#pragma unroll 8
  for (; w + 1 < nw; w += 2) {
    const double2 p = *reinterpret_cast<const double2 *>(r + w);
    s += p.x;
    s += p.y;
  }
  if (w < nw)
    s += r[w];
  return s;
}

// Block-level sum of K values; every thread receives the totals. Fixed order:
// butterfly inside each warp, then warps summed in index order. One lane per
// value sums the warps (all threads summing all values cost 2048 shared-memory
// reads per block for K = 8, more than the rest of the reduction).
template <int K>
KR_DEV void block_sum(TeamShared *sh, int &buf, double (&v)[K]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nw = (blockDim.x + 31) >> 5;
  double *r = sh->red[buf];
  if constexpr (K == 1) {
    const double t = warp_sum(v[0]);
    if (lane == 0)
      r[wid] = t;
    __syncthreads();
    v[0] = sum_warps(r, nw);
  } else {
    const double t = warp_sums<K>(v);
    if ((lane & (32 / K - 1)) == 0)
      r[(lane / (32 / K)) * KR_RED_LD + wid] = t;
    __syncthreads();
    const double s = lane < K ? sum_warps(r + lane * KR_RED_LD, nw) : 0.0;
#pragma unroll
    for (int k = 0; k < K; k++)
      v[k] = __shfl_sync(0xffffffffu, s, k);
  }
  buf ^= 1;
}

// ---------------------------------------------------------------------------
// Teams
// ---------------------------------------------------------------------------
struct TeamCta {
  TeamShared *sh;
  int *err; // per-solve status word (global)
  int buf;
  KR_DEV int64_t tid() const { return threadIdx.x; }
  KR_DEV int64_t nthreads() const { return blockDim.x; }
  KR_DEV int64_t warp_id() const { return threadIdx.x >> 5; }
  KR_DEV int64_t nwarps() const { return blockDim.x >> 5; }
  KR_DEV bool lead_cta() const { return true; }
  KR_DEV bool leader() const { return threadIdx.x == 0; }
  KR_DEV int cta_rank() const { return 0; }
  KR_DEV int ncta() const { return 1; }
  KR_DEV bool ok() const { return *(volatile int *)err == 0; }
  KR_DEV void sync() { __syncthreads(); }
  template <int K> KR_DEV void sum(double (&v)[K]) { block_sum<K>(sh, buf, v); }
  KR_DEV double sum1(double x) {
    double v[1] = {x};
    sum<1>(v);
    return v[0];
  }
  // h[q] = team total of this block's total s of value q (thread q < cnt); cnt <= KR_MDOT
  KR_DEV void dots(int cnt, double s, double *h) {
    if (threadIdx.x < (unsigned)cnt)
      h[threadIdx.x] = s;
  }
  // make values written by the leader block visible to the team
  KR_DEV void publish() { __syncthreads(); }
};

struct TeamGrid {
  TeamShared *sh;
  int *err;
  GridBarrierState *gb;
  double *gpart; // [2][gridDim.x][KR_MDOT]
  int buf;
  int gbuf;
  unsigned epoch = 0; // barriers reached
  KR_DEV int64_t tid() const { return (int64_t)blockIdx.x * blockDim.x + threadIdx.x; }
  KR_DEV int64_t nthreads() const { return (int64_t)gridDim.x * blockDim.x; }
  KR_DEV int64_t warp_id() const { return tid() >> 5; }
  KR_DEV int64_t nwarps() const { return nthreads() >> 5; }
  KR_DEV bool lead_cta() const { return blockIdx.x == 0; }
  KR_DEV bool leader() const { return blockIdx.x == 0 && threadIdx.x == 0; }
  KR_DEV int cta_rank() const { return blockIdx.x; }
  KR_DEV int ncta() const { return gridDim.x; }
  KR_DEV bool ok() const { return *(volatile int *)err == 0 && *(volatile int *)&gb->error == 0; }

  // Grid barrier with a bounded wait: one counter that only grows; barrier e is
  // passed when it reaches e times the blocks. On timeout it records
  // KRANS_ERR_TIMEOUT in the solve's status word; afterwards every barrier returns
  // immediately and the solver's bounded loops unwind. A counter that the last
  // block resets before it raises a generation costs two more trips to L2 (a solve of
  // 60013 incidence columns 72 ms, and 68 with this one); a count per block that all
  // blocks poll makes 148 x 148 polls contend (100 ms).
  KR_DEV void sync() {
    __syncthreads();
    epoch++;
    if (threadIdx.x == 0) {
      volatile int *verr = &gb->error;
      if (*verr == 0) {
        const unsigned want = epoch * gridDim.x;
        __threadfence();
        unsigned seen = atomicAdd(&gb->count, 1u) + 1u;
        // poll the counter alone; the error word and the clock are looked at once in
        // 64 polls (each costs a poll's time)
        const uint64_t t0 = globaltimer_ns();
        const uint64_t limit = gb->timeout_ns ? gb->timeout_ns : kBarrierTimeoutNs;
        for (unsigned polls = 1; (int)(seen - want) < 0; polls++) {
          asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&gb->count) : "memory");
          if (polls & 63)
            continue;
          if (*verr != 0)
            break;
          if (globaltimer_ns() - t0 > limit) {
            atomicCAS(&gb->error, 0, KRANS_ERR_TIMEOUT);
            atomicCAS(err, 0, KRANS_ERR_TIMEOUT);
            break;
          }
        }
        __threadfence();
      }
    }
    __syncthreads();
  }

  // sum over the blocks of partial `p` (stride KR_MDOT) by one warp, the same
  // fixed order in every block
  KR_DEV double sum_blocks(const double *p) const {
    double s = 0.0;
    for (unsigned b = threadIdx.x & 31; b < gridDim.x; b += 32)
      s += __ldcg(p + (size_t)b * KR_MDOT);
    return warp_sum(s);
  }
  template <int K> KR_DEV void sum(double (&v)[K]) {
    block_sum<K>(sh, buf, v);
    double *gp = gpart + (size_t)gbuf * gridDim.x * KR_MDOT;
    if (threadIdx.x == 0) {
#pragma unroll
      for (int k = 0; k < K; k++)
        gp[(size_t)blockIdx.x * KR_MDOT + k] = v[k];
    }
    sync();
    const int wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int k = wid; k < K; k += nw) {
      const double s = sum_blocks(gp + k);
      if ((threadIdx.x & 31) == 0)
        sh->bc[gbuf][k] = s;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; k++)
      v[k] = sh->bc[gbuf][k];
    gbuf ^= 1; // the next reduction writes the other slots, and the one after it is behind its barriers
  }
  KR_DEV void dots(int cnt, double s, double *h) {
    double *gp = gpart + (size_t)gbuf * gridDim.x * KR_MDOT;
    if (threadIdx.x < (unsigned)cnt)
      gp[(size_t)blockIdx.x * KR_MDOT + threadIdx.x] = s;
    sync();
    const int wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int q = wid; q < cnt; q += nw) {
      const double t = sum_blocks(gp + q);
      if ((threadIdx.x & 31) == 0)
        h[q] = t;
    }
    gbuf ^= 1;
  }
  KR_DEV double sum1(double x) {
    double v[1] = {x};
    sum<1>(v);
    return v[0];
  }
  KR_DEV void publish() { sync(); }
};

// A thread-block cluster (up to 16 blocks on distinct SMs of one GPC) as a
// team: hardware cluster barrier, reductions through distributed shared
// memory (each block writes its partials into every block's shared memory
// before the barrier, so that after it they are summed from local memory, in
// the order of the ranks).
struct TeamCluster {
  TeamShared *sh;
  int *err;
  int buf;
  int cbuf;
  unsigned rank, csize;
  KR_DEV int64_t tid() const { return (int64_t)rank * blockDim.x + threadIdx.x; }
  KR_DEV int64_t nthreads() const { return (int64_t)csize * blockDim.x; }
  KR_DEV int64_t warp_id() const { return tid() >> 5; }
  KR_DEV int64_t nwarps() const { return nthreads() >> 5; }
  KR_DEV bool lead_cta() const { return rank == 0; }
  KR_DEV bool leader() const { return rank == 0 && threadIdx.x == 0; }
  KR_DEV int cta_rank() const { return (int)rank; }
  KR_DEV int ncta() const { return (int)csize; }
  KR_DEV bool ok() const { return *(volatile int *)err == 0; }
  KR_DEV void sync() { cooperative_groups::this_cluster().sync(); }
  // The partials of one reduction go to buffer cbuf of every block; the next
  // reduction writes the other buffer, and the one after it is behind that
  // reduction's cluster barrier, which no block passes before it has read.
  template <int K> KR_DEV void sum(double (&v)[K]) {
    block_sum<K>(sh, buf, v);
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    if (threadIdx.x < csize) {
      double *peer = cl.map_shared_rank(&sh->cpart[cbuf][rank][0], threadIdx.x);
#pragma unroll
      for (int k = 0; k < K; k++)
        peer[k] = v[k];
    }
    cl.sync();
    double t[K];
#pragma unroll
    for (int k = 0; k < K; k++)
      t[k] = 0.0;
    for (unsigned r = 0; r < csize; r++) {
#pragma unroll
      for (int k = 0; k < K; k++)
        t[k] += sh->cpart[cbuf][r][k];
    }
#pragma unroll
    for (int k = 0; k < K; k++)
      v[k] = t[k];
    cbuf ^= 1;
  }
  KR_DEV void dots(int cnt, double s, double *h) {
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    if (threadIdx.x < (unsigned)cnt)
      for (unsigned r = 0; r < csize; r++)
        *cl.map_shared_rank(&sh->cpart[cbuf][rank][threadIdx.x], r) = s;
    cl.sync();
    if (threadIdx.x < (unsigned)cnt) {
      double t = 0.0;
      for (unsigned r = 0; r < csize; r++)
        t += sh->cpart[cbuf][r][threadIdx.x];
      h[threadIdx.x] = t;
    }
    cbuf ^= 1;
  }
  KR_DEV double sum1(double x) {
    double v[1] = {x};
    sum<1>(v);
    return v[0];
  }
  KR_DEV void publish() { sync(); }
};

// ---------------------------------------------------------------------------
// Element-wise team loops (grid-stride over the team's threads)
// ---------------------------------------------------------------------------
template <class Team, class F> KR_DEV void team_for(Team &tm, int64_t len, F f) {
  const int64_t nt = tm.nthreads();
  for (int64_t i = tm.tid(); i < len; i += nt)
    f(i);
}

template <class T> KR_DEV double to_d(T x) { return (double)x; }
KR_DEV int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }

template <class Team, class TX, class TY>
KR_DEV double team_dot(Team &tm, int64_t len, const TX *x, const TY *y) {
  double s = 0.0;
  const int64_t nt = tm.nthreads();
#pragma unroll 4
  for (int64_t i = tm.tid(); i < len; i += nt)
    s += to_d(x[i]) * to_d(y[i]);
  return tm.sum1(s);
}

template <class Team, class TX> KR_DEV double team_nrm2(Team &tm, int64_t len, const TX *x) {
  double s = 0.0;
  const int64_t nt = tm.nthreads();
  for (int64_t i = tm.tid(); i < len; i += nt) {
    const double v = to_d(x[i]);
    s += v * v;
  }
  return sqrt(tm.sum1(s));
}

// This thread's share of <S_k, w> for K columns of S (stride ld), two rows at
// a time: the 2 K + 2 loads are issued together before their products, which
// keeps enough of them in flight whatever the compiler makes of the loop (left
// to it, one build of the same source ran a Golub-Kahan step of 13877 incidence
// columns on two blocks in 150 us and the next in 190; this form takes 122).
// Columns from qn on repeat the last one (their sums are not used).
template <int K, class Team, class TS, class TW>
KR_DEV void dot_columns(Team &tm, int64_t len, const TS *S, int64_t ld, int qn, const TW *w, double (&acc)[K]) {
  const int64_t nt = tm.nthreads();
  const TS *col[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    acc[k] = 0.0;
    col[k] = S + (int64_t)min(k, qn - 1) * ld;
  }
  int64_t i = tm.tid();
  for (; i + nt < len; i += 2 * nt) {
    TS s0[K], s1[K];
    const TW w0 = w[i], w1 = w[i + nt];
#pragma unroll
    for (int k = 0; k < K; k++) {
      s0[k] = col[k][i];
      s1[k] = col[k][i + nt];
    }
    const double d0 = to_d(w0), d1 = to_d(w1);
#pragma unroll
    for (int k = 0; k < K; k++)
      acc[k] += to_d(s0[k]) * d0;
#pragma unroll
    for (int k = 0; k < K; k++)
      acc[k] += to_d(s1[k]) * d1;
  }
  if (i < len) {
    const double d0 = to_d(w[i]);
#pragma unroll
    for (int k = 0; k < K; k++)
      acc[k] += to_d(col[k][i]) * d0;
  }
}

// h[q] = <S_q, w> for q < ns (S columns at stride ld); results in tm.sh->h
// (all threads of every block see them after the call). Groups of 8 columns
// share one sweep over w; up to KR_MDOT columns share one team reduction (one
// per group, with every thread summing every value, made the Gram-Schmidt passes
// of small solves wait on reductions: a Golub-Kahan step of a 1000-unknown
// solve took 34 us, and takes 14).
template <class Team, class TS, class TW>
KR_DEV void team_multidot(Team &tm, int64_t len, const TS *S, int64_t ld, int ns, const TW *w) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  double *part = tm.sh->dots;
  for (int c0 = 0; c0 < ns; c0 += KR_MDOT) {
    const int cnt = min(KR_MDOT, ns - c0);
    for (int g = 0; g < cnt; g += KR_RED_K) {
      const int qn = min(KR_RED_K, cnt - g);
      const TS *Sg = S + (int64_t)(c0 + g) * ld;
      if (qn > KR_RED_K / 2) {
        double acc[KR_RED_K];
        dot_columns<KR_RED_K>(tm, len, Sg, ld, qn, w, acc);
        const double t = warp_sums<KR_RED_K>(acc);
        if ((lane & 3) == 0)
          part[(g + (lane >> 2)) * KR_RED_LD + wid] = t;
      } else {
        double acc[KR_RED_K / 2];
        dot_columns<KR_RED_K / 2>(tm, len, Sg, ld, qn, w, acc);
        const double t = warp_sums<KR_RED_K / 2>(acc);
        if ((lane & 7) == 0)
          part[(g + (lane >> 3)) * KR_RED_LD + wid] = t;
      }
    }
    __syncthreads();
    const double s = threadIdx.x < (unsigned)cnt ? sum_warps(part + threadIdx.x * KR_RED_LD, nw) : 0.0;
    tm.dots(cnt, s, tm.sh->h + c0);
    __syncthreads();
  }
}

// w -= sum_q S_q * coef[q]  (coef in shared memory). The subtractions run in
// q order for every element; the loads of several q are issued before their
// subtractions, so a thread keeps 8-16 loads in flight instead of waiting out
// one load per q (the short vectors of small solves are latency-bound on this).
template <class Team, class TS, class TW>
KR_DEV void team_multi_axpy(Team &tm, int64_t len, const TS *S, int64_t ld, int ns,
                            const double *coef, TW *w) {
  const int64_t nt = tm.nthreads();
  int64_t i = tm.tid();
  for (; i + 3 * nt < len; i += 4 * nt) {
    double acc[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      acc[u] = to_d(w[i + u * nt]);
    int q = 0;
    for (; q + 3 < ns; q += 4) {
      double sv[4][4];
#pragma unroll
      for (int t = 0; t < 4; t++)
#pragma unroll
        for (int u = 0; u < 4; u++)
          sv[t][u] = to_d(S[(int64_t)(q + t) * ld + i + u * nt]);
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const double cq = coef[q + t];
#pragma unroll
        for (int u = 0; u < 4; u++)
          acc[u] -= sv[t][u] * cq;
      }
    }
    for (; q < ns; q++) {
      const double cq = coef[q];
      const TS *sq = S + (int64_t)q * ld + i;
      double sv[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        sv[u] = to_d(sq[u * nt]);
#pragma unroll
      for (int u = 0; u < 4; u++)
        acc[u] -= sv[u] * cq;
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      w[i + u * nt] = (TW)acc[u];
  }
  for (; i < len; i += nt) {
    double acc = to_d(w[i]);
    int q = 0;
    for (; q + 7 < ns; q += 8) {
      double sv[8];
#pragma unroll
      for (int t = 0; t < 8; t++)
        sv[t] = to_d(S[(int64_t)(q + t) * ld + i]);
#pragma unroll
      for (int t = 0; t < 8; t++)
        acc -= sv[t] * coef[q + t];
    }
    for (; q < ns; q++)
      acc -= to_d(S[(int64_t)q * ld + i]) * coef[q];
    w[i] = (TW)acc;
  }
}

// Streams `len` elements with each thread handling 4 indices per step; the
// functor gets (index array, count) and must load all inputs before storing.
template <class Team, class F> KR_DEV void team_for4(Team &tm, int64_t len, F f) {
  const int64_t nt = tm.nthreads();
  int64_t i = tm.tid();
  for (; i + 3 * nt < len; i += 4 * nt) {
    const int64_t idx[4] = {i, i + nt, i + 2 * nt, i + 3 * nt};
    f(idx, 4);
  }
  for (; i < len; i += nt) {
    const int64_t idx[4] = {i, i, i, i};
    f(idx, 1);
  }
}

// ---------------------------------------------------------------------------
// CSR SpMV inside a team: `lanes` threads per row (power of two <= 32), rows
// handed out in warp-uniform blocks so the shuffles see full warps. The
// epilogue gets (row, sum) on the first lane of the row group.
// ---------------------------------------------------------------------------
template <class Acc> struct AccOf;
template <> struct AccOf<double> { using T = double; };
template <> struct AccOf<float> { using T = float; };

KR_DEV double2 ldg2(const double *a) { return __ldg(reinterpret_cast<const double2 *>(a)); }
KR_DEV float2 ldg2(const float *a) { return __ldg(reinterpret_cast<const float2 *>(a)); }

// Thread-per-row SpMV for matrices whose rows all hold exactly L = 1 or 2 entries
// (selections; incidence, shift and difference operators): no row pointers,
// vector loads of the (column, value) pairs, R rows in flight per thread. `pre`
// as in csr_mv_pre below.
template <int L, class Team, class VT, class GX, class Pre, class Epi>
KR_DEV void team_spmv_uniform(Team &tm, int64_t rows, const int32_t *__restrict__ ci,
                              const VT *__restrict__ val, GX gx, Pre pre, Epi epi) {
  static_assert(L == 1 || L == 2, "one or two entries");
  using Acc = typename AccOf<VT>::T;
  using XT = decltype(gx(0));
  using PT = decltype(pre(int64_t(0)));
  constexpr int R = KR_SPMV_ROWS;
  const int64_t nt = tm.nthreads();
  for (int64_t i0 = tm.tid(); i0 < rows; i0 += (int64_t)R * nt) {
    // rows past the end read the last row, so that all loads are unconditional
    int32_t c[R][L];
    VT v[R][L];
    PT pv[R];
#pragma unroll
    for (int u = 0; u < R; u++) {
      const int64_t i = imin64(i0 + (int64_t)u * nt, rows - 1);
      if constexpr (L == 2) {
        const int2 cc = __ldg(reinterpret_cast<const int2 *>(ci) + i);
        const auto vv = ldg2(val + 2 * i);
        c[u][0] = cc.x;
        c[u][1] = cc.y;
        v[u][0] = vv.x;
        v[u][1] = vv.y;
      } else {
        c[u][0] = __ldg(ci + i);
        v[u][0] = __ldg(val + i);
      }
      pv[u] = pre(i);
    }
    XT x[R][L];
#pragma unroll
    for (int u = 0; u < R; u++)
#pragma unroll
      for (int j = 0; j < L; j++)
        x[u][j] = gx(c[u][j]);
#pragma unroll
    for (int u = 0; u < R; u++) {
      const int64_t i = i0 + (int64_t)u * nt;
      Acc s = (Acc)v[u][0] * (Acc)x[u][0];
      if constexpr (L == 2)
        s += (Acc)v[u][1] * (Acc)x[u][1];
      if (i < rows)
        epi(i, s, pv[u]);
    }
  }
}

// CSR SpMV inside a team with a gather functor gx(col) for the input vector
// and a prologue pre(row) whose value goes to the epilogue epi(row, sum, value).
// The prologue loads what the epilogue combines with the row's sum (vectors at
// the row's index); it runs with the row pointers, so those loads overlap the
// gathers instead of following them.
// `lanes` threads per row (power of two <= 32), rows handed out in
// warp-uniform blocks so the shuffles see full warps; each warp walks R row
// groups at once (all row pointers, then all (column, value) pairs, then all
// gathers are issued before the FMAs). Lane `sub` of a row sums the entries
// b+sub, b+sub+lanes, ... in order, then a fixed butterfly combines the
// lanes: the result does not depend on R or on the team. The epilogue gets
// (row, sum) on the first lane of the row group.
template <class Team, class VT, class GX, class Pre, class Epi>
KR_DEV void team_spmv_lanes(Team &tm, int64_t rows, const int32_t *__restrict__ rp, const int32_t *__restrict__ ci,
                            const VT *__restrict__ val, GX gx, int lanes, Pre pre, Epi epi) {
  using Acc = typename AccOf<VT>::T;
  using XT = decltype(gx(0));
  using PT = decltype(pre(int64_t(0)));
  constexpr int R = KR_SPMV_ROWS;
  const int lane = threadIdx.x & 31;
  const int sub = lane & (lanes - 1), grp = lane / lanes;
  const int rpw = 32 / lanes;
  const int64_t chunk = (int64_t)rpw * R;
  const int64_t nw = tm.nwarps();
  for (int64_t base = tm.warp_id() * chunk; base < rows; base += nw * chunk) {
    int32_t b[R], e[R];
    PT pv[R];
#pragma unroll
    for (int u = 0; u < R; u++) {
      const int64_t i = base + (int64_t)u * rpw + grp;
      b[u] = 0;
      e[u] = 0;
      if (i < rows) {
        b[u] = __ldg(rp + i) + sub;
        e[u] = __ldg(rp + i + 1);
        if (sub == 0)
          pv[u] = pre(i);
      }
    }
    Acc s[R];
#pragma unroll
    for (int u = 0; u < R; u++)
      s[u] = Acc(0);
    for (int32_t j = 0;; j += lanes) {
      int32_t c[R];
      VT v[R];
      bool ok[R], more = false;
#pragma unroll
      for (int u = 0; u < R; u++) {
        const int32_t k = b[u] + j;
        ok[u] = k < e[u];
        more |= (k + lanes) < e[u];
        c[u] = ok[u] ? __ldg(ci + k) : 0;
        v[u] = ok[u] ? __ldg(val + k) : VT(0);
      }
      XT xv[R];
#pragma unroll
      for (int u = 0; u < R; u++)
        xv[u] = ok[u] ? gx(c[u]) : XT(0);
#pragma unroll
      for (int u = 0; u < R; u++)
        if (ok[u])
          s[u] += (Acc)v[u] * (Acc)xv[u];
      if (!more)
        break;
    }
#pragma unroll
    for (int u = 0; u < R; u++) {
      for (int o = lanes >> 1; o > 0; o >>= 1)
        s[u] += __shfl_xor_sync(0xffffffffu, s[u], o);
      const int64_t i = base + (int64_t)u * rpw + grp;
      if (i < rows && sub == 0)
        epi(i, s[u], pv[u]);
    }
  }
}

// CSR SpMV on sorted slices (SlicedView): a warp takes a slice of 32 rows of
// nearly equal length, one row per lane; round j of a slice holds entry j of
// each of its rows, padded with zero values, so a round's columns and values
// are one coalesced read at a known place. Rows are summed in storage order by
// one lane: no shuffles, and the same sum whatever the team. The prologue and
// epilogue get the row and its slot (position in the sorted order): vectors
// private to a loop can be kept by slot and read coalesced.
// A warp gathers J rounds at a time and reads the following J (of the slice, or
// of its next one) before it sums them. Row-major entries (team_spmv_lanes)
// cost a sector lookup per row and load; F^T of an incidence matrix (4000 rows
// of 6 entries on average) takes 47,500 SM cycles there and 24,800 here. J = 2,
// 4, 6: 29,000, 22,500, 25,900 with the vectors in shared memory.
template <class Team, class VT, class GX, class Pre, class Epi>
KR_DEV void team_spmv_sliced(Team &tm, const SlicedView &S, const VT *__restrict__ sval, GX gx, Pre pre, Epi epi) {
  using Acc = typename AccOf<VT>::T;
  using XT = decltype(gx(0));
  using PT = decltype(pre(0, 0));
  constexpr int J = KR_SLICE_J;
  const int lane = threadIdx.x & 31;
  const int nsl = S.slices, nw = (int)tm.nwarps();
  const int32_t *__restrict__ off = S.off, *__restrict__ rowmap = S.row, *__restrict__ sci = S.ci;
  int sl = (int)tm.warp_id();
  if (sl >= nsl)
    return;
  int32_t c[J];
  VT v[J];
  auto fetch = [&](int32_t o, int32_t oe, int32_t(&c)[J], VT(&v)[J]) {
    const int32_t *pc = sci + (size_t)o * 32 + lane;
    const VT *pvv = sval + (size_t)o * 32 + lane;
#pragma unroll
    for (int q = 0; q < J; q++) {
      c[q] = o + q < oe ? __ldg(pc + q * 32) : 0;
      v[q] = o + q < oe ? __ldg(pvv + q * 32) : VT(0);
    }
  };
  int32_t o = __ldg(off + sl), oe = __ldg(off + sl + 1);
  int row = __ldg(rowmap + sl * 32 + lane);
  fetch(o, oe, c, v);
  // slices ahead: bounds and rows of the next two, prologue of the next one
  // (past the end: the last slice again, unused)
  int nx = min(sl + nw, nsl - 1);
  int32_t on = __ldg(off + nx), oen = __ldg(off + nx + 1);
  int rown = __ldg(rowmap + nx * 32 + lane);
  PT pv = pre(max(row, 0), sl * 32 + lane);
  int n2 = min(sl + 2 * nw, nsl - 1);
  int32_t o_2 = __ldg(off + n2), oe_2 = __ldg(off + n2 + 1);
  int row_2 = __ldg(rowmap + n2 * 32 + lane);
  Acc s = Acc(0);
  for (;;) {
    XT x[J];
#pragma unroll
    for (int q = 0; q < J; q++)
      x[q] = o + q < oe ? gx(c[q]) : XT(0);
    const bool more = o + J < oe; // the slice goes on
    const int32_t on1 = more ? o + J : on, oe1 = more ? oe : oen;
    int32_t cn[J];
    VT vn[J];
    fetch(on1, oe1, cn, vn);
#pragma unroll
    for (int q = 0; q < J; q++)
      s += (Acc)v[q] * (Acc)x[q];
    if (!more) {
      const PT pn = pre(max(rown, 0), nx * 32 + lane);
      if (row >= 0)
        epi(row, sl * 32 + lane, s, pv);
      sl += nw;
      if (sl >= nsl)
        break;
      s = Acc(0);
      pv = pn;
      row = rown;
      on = o_2;
      oen = oe_2;
      rown = row_2;
      nx = n2;
      n2 = min(sl + 2 * nw, nsl - 1);
      o_2 = __ldg(off + n2);
      oe_2 = __ldg(off + n2 + 1);
      row_2 = __ldg(rowmap + n2 * 32 + lane);
    }
    o = on1;
    oe = oe1;
#pragma unroll
    for (int q = 0; q < J; q++) {
      c[q] = cn[q];
      v[q] = vn[q];
    }
  }
}

template <class VT> KR_DEV const VT *csr_values(const CsrView &V) {
  if constexpr (sizeof(VT) == 8)
    return V.v64;
  else
    return V.v32;
}
template <class VT> KR_DEV const VT *sliced_values(const SlicedView &S) {
  if constexpr (sizeof(VT) == 8)
    return S.v64;
  else
    return S.v32;
}

// y = V x with VT values, gather gx(col), prologue pre(row, slot) and epilogue
// epi(row, slot, sum, prologue's value). Operands with sorted slices: those (see
// pick_slices); rows of exactly 1 or 2 entries: vector loads, no row pointers; else
// `lanes` threads per row (slot = row in both).
template <class VT, class Team, class GX, class Pre, class Epi>
KR_DEV void csr_mv_pre(Team &tm, const CsrView &V, GX gx, Pre pre, Epi epi) {
  using Acc = typename AccOf<VT>::T;
  if (V.sl.slices) {
    team_spmv_sliced(tm, V.sl, sliced_values<VT>(V.sl), gx, pre, epi);
    return;
  }
  auto pre1 = [&](int64_t i) { return pre((int)i, (int)i); };
  auto epi1 = [&](int64_t i, Acc s, decltype(pre(0, 0)) p) { epi((int)i, (int)i, s, p); };
  if (V.ulen == 2)
    team_spmv_uniform<2>(tm, V.rows, V.ci, csr_values<VT>(V), gx, pre1, epi1);
  else if (V.ulen == 1)
    team_spmv_uniform<1>(tm, V.rows, V.ci, csr_values<VT>(V), gx, pre1, epi1);
  else
    team_spmv_lanes(tm, V.rows, V.rp, V.ci, csr_values<VT>(V), gx, V.lanes, pre1, epi1);
}
// the same from a plain vector and without a prologue: epi(row, sum)
struct NoPrologue {
  KR_DEV char operator()(int64_t) const { return 0; }
  KR_DEV char operator()(int, int) const { return 0; }
};
template <class VT, class Team, class XT, class Epi>
KR_DEV void csr_mv(Team &tm, const CsrView &V, const XT *x, Epi epi) {
  using Acc = typename AccOf<VT>::T;
  csr_mv_pre<VT>(
      tm, V, [&](int32_t c) { return x[c]; }, NoPrologue(), [&](int i, int, Acc s, char) { epi(i, s); });
}

// CSR SpMV over KR_NBP right-hand sides stored interleaved (element (i, j) at
// i * KR_NBP + j). Eight consecutive threads share a row and thread j of the
// group owns column j (the team size is a multiple of KR_NBP, so a thread's
// column never changes): the (column, value) loads are broadcast inside the
// group and the gather reads 64 contiguous bytes per entry. Each thread sums
// its column over the row's entries in storage order (the same order in both
// variants below); threads whose column is not `active` skip the row. Every
// thread keeps R rows in flight so the gathers of several rows overlap.
template <int L, int R, class Team, class GX, class Epi>
KR_DEV void team_spmv_block_uniform(Team &tm, int64_t rows, const int32_t *__restrict__ ci,
                                    const double *__restrict__ val, GX gx, Epi epi) {
  const int64_t ng = tm.nthreads() / KR_NBP;
  for (int64_t i0 = tm.tid() / KR_NBP; i0 < rows; i0 += (int64_t)R * ng) {
    int32_t c[R][L];
    double v[R][L];
#pragma unroll
    for (int u = 0; u < R; u++) {
      const int64_t i = i0 + (int64_t)u * ng;
#pragma unroll
      for (int j = 0; j < L; j++) {
        c[u][j] = i < rows ? __ldg(ci + i * L + j) : 0;
        v[u][j] = i < rows ? __ldg(val + i * L + j) : 0.0;
      }
    }
    double xv[R][L];
#pragma unroll
    for (int u = 0; u < R; u++)
#pragma unroll
      for (int j = 0; j < L; j++)
        xv[u][j] = i0 + (int64_t)u * ng < rows ? gx(c[u][j]) : 0.0;
#pragma unroll
    for (int u = 0; u < R; u++) {
      const int64_t i = i0 + (int64_t)u * ng;
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < L; j++)
        s += v[u][j] * xv[u][j];
      if (i < rows)
        epi(i, s);
    }
  }
}

template <class Team, class GX, class Epi>
KR_DEV void team_spmv_block(Team &tm, int64_t rows, const int32_t *__restrict__ rp,
                            const int32_t *__restrict__ ci, const double *__restrict__ val, int32_t ulen,
                            bool active, GX gx, Epi epi) {
  if (!active)
    return; // no barrier inside: threads of inactive columns simply skip
  if (ulen == 2) {
    team_spmv_block_uniform<2, 4>(tm, rows, ci, val, gx, epi);
    return;
  }
  if (ulen == 1) {
    team_spmv_block_uniform<1, 8>(tm, rows, ci, val, gx, epi);
    return;
  }
  if (ulen == 4) {
    team_spmv_block_uniform<4, 2>(tm, rows, ci, val, gx, epi);
    return;
  }
  constexpr int R = 4;
  const int64_t ng = tm.nthreads() / KR_NBP;
  for (int64_t i0 = tm.tid() / KR_NBP; i0 < rows; i0 += (int64_t)R * ng) {
    int32_t b[R], e[R];
#pragma unroll
    for (int u = 0; u < R; u++) {
      const int64_t i = i0 + (int64_t)u * ng;
      b[u] = 0;
      e[u] = 0;
      if (i < rows) {
        b[u] = __ldg(rp + i);
        e[u] = __ldg(rp + i + 1);
      }
    }
    double s[R];
#pragma unroll
    for (int u = 0; u < R; u++)
      s[u] = 0.0;
    for (int32_t j = 0;; ++j) {
      int32_t c[R];
      double v[R];
      bool ok[R], more = false;
#pragma unroll
      for (int u = 0; u < R; u++) {
        const int32_t k = b[u] + j;
        ok[u] = k < e[u];
        more |= (k + 1) < e[u];
        c[u] = ok[u] ? __ldg(ci + k) : 0;
        v[u] = ok[u] ? __ldg(val + k) : 0.0;
      }
      double xv[R];
#pragma unroll
      for (int u = 0; u < R; u++)
        xv[u] = ok[u] ? gx(c[u]) : 0.0;
#pragma unroll
      for (int u = 0; u < R; u++)
        if (ok[u])
          s[u] += v[u] * xv[u];
      if (!more)
        break;
    }
#pragma unroll
    for (int u = 0; u < R; u++) {
      const int64_t i = i0 + (int64_t)u * ng;
      if (i < rows)
        epi(i, s[u]);
    }
  }
}

// Algorithmic HBM bytes of one CSR SpMV (rows r, cols c, nnz z, value width
// w, x width wx, y width wy): row pointers, columns+values, x once, y once.
__host__ __device__ inline double spmv_bytes(int64_t r, int64_t c, int64_t z, int w, int wx, int wy) {
  return 4.0 * (double)(r + 1) + (double)z * (w + 4) + (double)c * wx + (double)r * wy;
}

// ---------------------------------------------------------------------------
// Random normal vectors
// ---------------------------------------------------------------------------
KR_DEV uint32_t mt_temper(uint32_t y) {
  y ^= y >> 11;
  y ^= (y << 7) & 0x9d2c5680u;
  y ^= (y << 15) & 0xefc60000u;
  y ^= y >> 18;
  return y;
}

KR_DEV uint32_t mt_twist(uint32_t a, uint32_t b) {
  return (((a & 0x80000000u) | (b & 0x7fffffffu)) >> 1) ^ (b & 1u ? 0x9908b0dfu : 0u);
}
// Word i of the state that follows `src`. The recurrence new[i] = x[i + 397] ^
// twist(old[i], old[i + 1]) reads a new word from i = 227 on; those are written
// out in terms of old words (one twist more from 227 on, two from 454 on), so all
// words are independent. Loads and twists that word i does not need are made on
// some other word and dropped, so that the loads go out together.
KR_DEV uint32_t mt_next_word(const uint32_t *src, int i) {
  const int j = i >= 227 ? i - 227 : 0, k = i >= 454 ? i - 454 : 0;
  const uint32_t far = src[i < 227 ? i + 397 : i < 454 ? i + 170 : i - 57];
  const uint32_t a0 = src[i], a1 = src[i < 623 ? i + 1 : 0], b0 = src[j], b1 = src[j + 1], c0 = src[k], c1 = src[k + 1];
  const uint32_t new0 = src[397] ^ mt_twist(src[0], src[1]); // follows the last old word
  uint32_t v = far ^ mt_twist(a0, i < 623 ? a1 : new0);
  v ^= i >= 227 ? mt_twist(b0, b1) : 0u;
  v ^= i >= 454 ? mt_twist(c0, c1) : 0u;
  return v;
}
// MT19937 regeneration of 624 words by a block: src -> dst, no barrier inside
KR_DEV void mt_regen_block(const uint32_t *src, uint32_t *dst) {
  for (int i = threadIdx.x; i < 624; i += blockDim.x)
    dst[i] = mt_next_word(src, i);
}

// One polar attempt from four words (two 53-bit canonicals): the point (x, y)
// and its squared radius; true if it is accepted.
KR_DEV bool polar_attempt(const uint32_t *w, double &x, double &y, double &r2) {
  const double a = (double)mt_temper(w[0]), b = (double)mt_temper(w[1]);
  const double c = (double)mt_temper(w[2]), d = (double)mt_temper(w[3]);
  double u1 = __dadd_rn(a, __dmul_rn(b, 4294967296.0)) * 0x1p-64;
  double u2 = __dadd_rn(c, __dmul_rn(d, 4294967296.0)) * 0x1p-64;
  if (u1 >= 1.0)
    u1 = 0x1.fffffffffffffp-1;
  if (u2 >= 1.0)
    u2 = 0x1.fffffffffffffp-1;
  x = __dadd_rn(__dmul_rn(2.0, u1), -1.0);
  y = __dadd_rn(__dmul_rn(2.0, u2), -1.0);
  r2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
  return !(r2 > 1.0 || r2 == 0.0);
}
// an accepted point's scale: the normals are y times it, then x times it
KR_DEV double polar_scale(double r2) { return sqrt(-2.0 * log(r2) / r2); }

// One block draws the next n normals of an MT19937 + polar stream, exactly
// as std::normal_distribution<double> consumes std::mt19937 in libstdc++:
// each polar attempt takes four 32-bit words (two 53-bit canonicals); an
// accepted attempt yields y*m then x*m, and an unused x*m is carried over.
// `ring` holds nblk states of 624 words in shared memory; a round generates
// them one after the other and takes one attempt per thread from all of them
// (needs blockDim.x >= 156 nblk). Bound by the barriers between dependent
// states and by one SM's FP64 rate in log and square root.
KR_DEV void block_mt_normals(RngState *st, double *out, int64_t n, uint32_t *ring, int nblk) {
  __shared__ int s_wsum[KR_MAX_WARPS];
  __shared__ int s_last;
  __shared__ double s_saved;
  __shared__ int s_has_saved;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = (blockDim.x + 31) >> 5;
  for (int i = t; i < 624; i += blockDim.x)
    ring[i] = st->mt[i];
  int idx = st->idx; // first unused word of the ring
  if (t == 0) {
    s_has_saved = st->has_saved;
    s_saved = st->saved;
    s_last = -1;
  }
  __syncthreads();
  int64_t pos = 0;
  if (n > 0 && s_has_saved) {
    if (t == 0)
      out[0] = s_saved;
    pos = 1;
    __syncthreads();
    if (t == 0)
      s_has_saved = 0;
  }
  __syncthreads();
  for (bool first = true; pos < n; first = false) {
    // the states after the last one; it becomes the first of the ring
    if (!first) {
      mt_regen_block(ring + (nblk - 1) * 624, ring);
      idx = 0;
      __syncthreads();
    }
    for (int b = 1; b < nblk; b++) {
      mt_regen_block(ring + (b - 1) * 624, ring + b * 624);
      __syncthreads();
    }
    const int navail = (nblk * 624 - idx) >> 2;
    double x = 0.0, y = 0.0, r2 = 0.0;
    const bool acc = t < navail && polar_attempt(ring + idx + 4 * t, x, y, r2);
    const unsigned bal = __ballot_sync(0xffffffffu, acc);
    if (lane == 0)
      s_wsum[wid] = __popc(bal);
    __syncthreads();
    const int mine = lane < nw ? s_wsum[lane] : 0;
    const int before = __reduce_add_sync(0xffffffffu, lane < wid ? mine : 0) + __popc(bal & ((1u << lane) - 1u));
    const int total = __reduce_add_sync(0xffffffffu, mine);
    const int64_t need = (n - pos + 1) >> 1; // pairs still needed
    if (acc && before < need) {
      const double mult = polar_scale(r2);
      const int64_t p = pos + 2 * (int64_t)before;
      out[p] = __dmul_rn(y, mult);
      if (p + 1 < n) {
        out[p + 1] = __dmul_rn(x, mult);
      } else {
        s_saved = __dmul_rn(x, mult);
        s_has_saved = 1;
      }
      if (before == need - 1)
        s_last = t;
    }
    __syncthreads();
    if (total >= need) {
      idx += 4 * (s_last + 1);
      pos = n;
    } else {
      idx = nblk * 624;
      pos += 2 * (int64_t)total;
    }
  }
  // the state that holds the last used word (an exhausted state stays, as the
  // next draw regenerates it), and the next word in it
  const int last = idx > 624 ? (idx - 1) / 624 : 0;
  for (int i = t; i < 624; i += blockDim.x)
    st->mt[i] = ring[last * 624 + i];
  if (t == 0) {
    st->idx = idx - last * 624;
    st->has_saved = s_has_saved;
    st->saved = s_saved;
  }
  __syncthreads();
}

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw: "Parallel random numbers: as
// easy as 1, 2, 3", SC'11), counter-based.
KR_DEV uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
  for (int r = 0; r < 10; r++) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}

// Normal variate number `ctr` of the stream `key` (Box-Muller on two
// 53-bit uniforms from one Philox block).
KR_DEV double philox_normal(uint64_t key, uint64_t ctr) {
  const uint4 r = philox4x32_10(make_uint4((uint32_t)ctr, (uint32_t)(ctr >> 32), 0x4b52414eu, 0u),
                                make_uint2((uint32_t)key, (uint32_t)(key >> 32)));
  const uint64_t a = ((uint64_t)r.x << 21) ^ (uint64_t)(r.y >> 11);
  const uint64_t b = ((uint64_t)r.z << 21) ^ (uint64_t)(r.w >> 11);
  const double u1 = ((double)(a & ((1ull << 53) - 1)) + 1.0) * 0x1p-53; // (0, 1]
  const double u2 = (double)(b & ((1ull << 53) - 1)) * 0x1p-53;         // [0, 1)
  return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}

// Fill out[0..n) with the stream's next n normals, as a team. MT19937 is
// generated by the team's leader block; Philox by every thread.
template <class Team> KR_DEV void team_random_normal(Team &tm, RngState *st, double *out, int64_t n) {
  if (*(volatile int32_t *)&st->mode == KRANS_RNG_PHILOX) {
    const uint64_t key = *(volatile uint64_t *)&st->philox_key;
    const uint64_t base = *(volatile uint64_t *)&st->philox_ctr;
    team_for(tm, n, [&](int64_t i) { out[i] = philox_normal(key, base + (uint64_t)i); });
    tm.sync();
    if (tm.leader())
      st->philox_ctr = base + (uint64_t)n;
    tm.publish();
  } else {
    // the ring takes the space of team_multidot's partials (3 states on 512 threads)
    static_assert(sizeof(TeamShared::dots) >= 3 * 624 * 4, "ring of MT19937 states");
    if (tm.lead_cta())
      block_mt_normals(st, out, n, reinterpret_cast<uint32_t *>(tm.sh->dots), 3);
    tm.publish();
  }
}

} // namespace kr
