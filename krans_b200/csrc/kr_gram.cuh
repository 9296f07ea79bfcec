// Tall-skinny products of the block solver, on the FP64 tensor cores:
//   team_tn_panels:     S = Z^T Z with G = Z^T (AZ), or C = A^T B: shared-memory
//                       panels, for long, wide blocks
//   team_tn_direct:     the same for short or narrow blocks, one warp per output
//                       tile
//   team_gemm_nn:       out (-)= Z * Y[roff:roff+zc, 0:q] (n x q), shared-memory
//                       chunks (team_combine, team_combine_sub)
// Sums run in a fixed order that depends only on the team size, so results
// are deterministic for a given team size.
#pragma once

#include "kr_device.cuh"

namespace kr {

// FP64 tensor-core MMA (DMMA) m8n8k4: D = A(8x4, row) * B(4x8, col) + C.
KR_DEV void dmma_8x8x4(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// f(e, sum over the team's blocks of part[rank * stride + e]) for e < count,
// with two sums when `two` (the second at offset `second`). Few blocks: a thread
// per element, blocks in order. Many: a warp per element, each lane over its
// share of the blocks and a butterfly (one thread summing 148 partials waits
// out 148 loads).
template <class Team, class F>
KR_DEV void team_sum_ranks(Team &tm, int64_t count, const double *part, size_t stride, size_t second, F f) {
  const int ncta = tm.ncta();
  if (ncta < 32) {
    for (int64_t e = tm.tid(); e < count; e += tm.nthreads()) {
      double s = 0.0, g = 0.0;
      for (int r = 0; r < ncta; r++) {
        s += __ldcg(part + (size_t)r * stride + e);
        if (second)
          g += __ldcg(part + (size_t)r * stride + second + e);
      }
      f(e, s, g);
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  for (int64_t e = tm.warp_id(); e < count; e += tm.nwarps()) {
    double s = 0.0, g = 0.0;
    for (int r = lane; r < ncta; r += 32) {
      s += __ldcg(part + (size_t)r * stride + e);
      if (second)
        g += __ldcg(part + (size_t)r * stride + second + e);
    }
    s = warp_sum(s);
    if (second)
      g = warp_sum(g);
    if (lane == 0)
      f(e, s, g);
  }
}

// Rows [r0, r1) of an 8 x 8 tile of X^T Y (and of X^T W when TWO) by one warp,
// operands straight from global memory; xa, yb, wb: this lane's column, or
// nullptr past the last one. Four steps of four rows are loaded together. The
// MMA lane layout of m8n8k4: A(row = lane >> 2, k = lane & 3), B(k = lane & 3,
// col = lane >> 2), C rows lane >> 2, columns 2 (lane & 3) and the next.
template <bool TWO>
KR_DEV void warp_tn_tile(int64_t r0, int64_t r1, const double *xa, const double *yb, const double *wb, double (&s)[2],
                         double (&g)[2]) {
  constexpr int U = 4;
  const int k = threadIdx.x & 3;
  double cs[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, cg[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int64_t base = r0; base < r1; base += 4 * U) { // warp-uniform trip count
    double x[U], y[U], w[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int64_t r = base + 4 * u + k;
      const bool in = r < r1;
      x[u] = in && xa ? xa[r] : 0.0;
      y[u] = in && yb ? yb[r] : 0.0;
      if constexpr (TWO)
        w[u] = in && wb ? wb[r] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      dmma_8x8x4(cs[u & 1][0], cs[u & 1][1], x[u], y[u]);
      if constexpr (TWO)
        dmma_8x8x4(cg[u & 1][0], cg[u & 1][1], x[u], w[u]);
    }
  }
#pragma unroll
  for (int h = 0; h < 2; h++) {
    s[h] = cs[0][h] + cs[1][h];
    g[h] = cg[0][h] + cg[1][h];
  }
}

// The direct forms, for short or narrow blocks: each block reduces its fixed
// row range into a private partial, 8 x 8 tiles by warps; with fewer tiles than
// warps the rows are split among the warps too, whose pieces are added in order
// in shared memory. The blocks' partials are summed in a fixed order. Bound by the
// latency of dependent steps of 4 to 16 rows (a block of 148 has 338 of 50021
// rows); the Gram pairs of that LOBPCG solve (36 and 12 columns) took 9.8 ms in
// all and take 4.5, its orthonormalisations 53 and 41 ms.
//   SYM: S = Z^T Z and G = Z^T W (p x p): like the reference's form_gram
//        (LOBPCGSolver.cpp:67-80), which sets S(i,j) = S(j,i) = Z_i.Z_j and
//        G(i,j) = G(j,i) = Z_i.(AZ)_j for i <= j, only the upper triangles are
//        formed and then mirrored; `part` holds 2 p^2 doubles a block
//   else: S = Z^T W (p x q); p q doubles a block
template <bool SYM, class Team>
KR_DEV void team_tn_direct(Team &tm, int64_t n, const double *Z, int p, const double *W, int q, int64_t ld, double *S,
                           double *G, double *part) {
  constexpr int TILE = SYM ? 128 : 64; // doubles of a tile's piece
  const int tp = (p + 7) / 8, tq = (q + 7) / 8, ntiles = SYM ? tp * (tp + 1) / 2 : tp * tq;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int ncta = tm.ncta(), rank = tm.cta_rank();
  const int64_t per = (n + ncta - 1) / ncta;
  const int64_t r0 = imin64((int64_t)rank * per, n), r1 = imin64(r0 + per, n);
  const size_t stride = (SYM ? 2 : 1) * (size_t)p * q;
  double *my = part + (size_t)rank * stride;
  double *pieces = tm.sh->dots; // (slab, tile) pieces, ntiles nslab <= pieces that fit
  constexpr int fit = KR_MDOT * KR_RED_LD / TILE;
  const int nslab = max(1, min(nw, fit) / ntiles);
  const int64_t slab_rows = kr_round_up((r1 - r0 + nslab - 1) / nslab, 16);
  for (int t = wid; t < ntiles * nslab; t += nw) {
    const int tile = t % ntiles, slab = t / ntiles;
    int bi = tile % tp, bj = tile / tp;
    if (SYM) { // upper-triangular tile index -> bi <= bj
      bi = 0;
      int rem = tile;
      while (rem >= tp - bi) {
        rem -= tp - bi;
        bi++;
      }
      bj = bi + rem;
    }
    const int ia = bi * 8 + (lane >> 2), jb = bj * 8 + (lane >> 2);
    const double *xa = ia < p ? Z + (int64_t)ia * ld : nullptr;
    const double *yb = jb < q ? (SYM ? Z : W) + (int64_t)jb * ld : nullptr;
    const double *wb = SYM && jb < q ? W + (int64_t)jb * ld : nullptr;
    const int64_t s0 = imin64(r0 + slab * slab_rows, r1), s1 = imin64(s0 + slab_rows, r1);
    double s[2], g[2];
    warp_tn_tile<SYM>(s0, s1, xa, yb, wb, s, g);
    const int ci = lane >> 2, cj = 2 * (lane & 3);
    if (nslab > 1) {
      double *pc = pieces + t * TILE;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        pc[ci + 8 * (cj + h)] = s[h];
        if (SYM)
          pc[64 + ci + 8 * (cj + h)] = g[h];
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int i = bi * 8 + ci, j = bj * 8 + cj + h;
        if (i < p && j < q) {
          my[i + (size_t)j * p] = s[h];
          if (SYM)
            my[(size_t)p * q + i + (size_t)j * p] = g[h];
        }
      }
    }
  }
  if (nslab > 1) {
    __syncthreads();
    for (int e = threadIdx.x; e < p * q; e += blockDim.x) {
      const int i = e % p, j = e / p, bi = i / 8, bj = j / 8;
      if (SYM && bi > bj)
        continue;
      const int tile = SYM ? bi * tp - bi * (bi - 1) / 2 + (bj - bi) : bj * tp + bi;
      double s = 0.0, g = 0.0;
      for (int k = 0; k < nslab; k++) {
        const double *pc = pieces + (k * ntiles + tile) * TILE + (i & 7) + 8 * (j & 7);
        s += pc[0];
        if (SYM)
          g += pc[64];
      }
      my[e] = s;
      if (SYM)
        my[(size_t)p * q + e] = g;
    }
  }
  tm.sync();
  team_sum_ranks(tm, (int64_t)p * q, part, stride, SYM ? (size_t)p * q : 0, [&](int64_t e, double s, double g) {
    if (!SYM) {
      S[e] = s;
      return;
    }
    const int j = (int)(e / p), i = (int)(e % p);
    if (i > j)
      return;
    S[i + (size_t)j * p] = s;
    S[j + (size_t)i * p] = s;
    G[i + (size_t)j * p] = g;
    G[j + (size_t)i * p] = g;
  });
  tm.sync();
}

#define KR_TN_ROWS 131072 // rows from which the panel form of the A^T B products runs
#define KR_TN_COLS 32     // and columns

// ---- panel products -----------------------------------------------------------
// Asynchronous copies into the shared-memory panels: `live` of the W doubles
// (W = 1 or 2) from global memory, zeros for the rest.
template <int W> KR_DEV void cp_async_f64(double *dst, const double *src, int live) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if constexpr (W == 2)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(8 * live) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(8 * live) : "memory");
}
KR_DEV void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> KR_DEV void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
KR_DEV bool aligned16(const double *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Products of tall blocks over their rows, on the FP64 tensor cores:
//   SYM:  S = Z^T Z and, when W is given, G = Z^T W (p x p): only the upper 64
//         x 64 tiles are formed, and mirrored, as the reference's form_gram does
//         (LOBPCGSolver.cpp:67-80: S(i,j) = S(j,i) = Z_i.Z_j, G(i,j) = G(j,i) =
//         Z_i.(AZ)_j for i <= j);
//   else: S = Z^T W (p x q).
// Work items are (tile, chunk of rows). A block stages 32-row panels of the
// tile's columns of Z (and W) in shared memory, the next panel on its way by
// cp.async while one is multiplied; each of its 16 warps accumulates a 16 x 16 piece of S and of G (2 x
// 2 DMMA 8x8 tiles each) and skips pieces below the diagonal or past the last
// column. Partial tiles are summed in chunk order, so the result depends only
// on the team size.
// Bound by the DMMA pipe (36.9 TFLOP/s measured). The panel pitch of 36 doubles
// puts the 8 x 4 fragment of a DMMA on distinct banks (33 cost four-way
// conflicts and held the kernel to 11 TFLOP/s executed), and the pieces are
// dealt to the warps so that the ones past an edge do not all fall to one of
// the SM's four pipes. The chunk count fills two rounds of the team's blocks,
// not a little more than two. At n = 4194304, counting 2 n p^2 a product: S and
// G of p = 288 17.6 -> 35.5 TFLOP/s, of p = 96 9.8 -> 26.1; a 64 x 96
// projection 11.4 -> 19.0. Narrow blocks on many thread blocks stay with the
// direct forms: p = 36 at n = 50021 took 0.10 ms there and 0.16 ms in panels.
// `part` must hold (2 ncta + tiles) * 4096 doubles, twice that with SYM; needs
// 512 threads and tn_panel_smem_bytes() of dynamic shared memory.
#define KR_GT 64 // tile edge
#define KR_GP 32 // rows per panel
#define KR_GL 36 // panel pitch
#define KR_GS 2  // panels held: one multiplied, one on its way
__host__ __device__ constexpr size_t tn_panel_smem_bytes() { return (size_t)KR_GS * 3 * KR_GT * KR_GL * 8; }

template <bool SYM, class Team>
KR_DEV void team_tn_panels(Team &tm, int64_t n, const double *Z, int p, const double *W, int q, int64_t ld, double *S,
                           double *G, double *part) {
  extern __shared__ __align__(16) double kr_gemm_smem[];
  constexpr int PANEL = KR_GT * KR_GL, STAGE = 3 * PANEL;
  constexpr int ITEM = (SYM ? 2 : 1) * KR_GT * KR_GT;
  const bool two = SYM && W != nullptr; // S and G
  const int tp = (p + KR_GT - 1) / KR_GT, tq = (q + KR_GT - 1) / KR_GT;
  const int tiles = SYM ? tp * (tp + 1) / 2 : tp * tq;
  const int ncta = tm.ncta();
  const int64_t kblocks = (n + KR_GP - 1) / KR_GP;
  const int nch = (int)imin64(kblocks, 2 * ncta / tiles);
  const int nchunks = nch > 0 ? nch : 1;
  const int64_t kb_per = (kblocks + nchunks - 1) / nchunks; // panels per chunk
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int wr = (wid >> 2) * 16, wc = ((wid + (wid >> 2)) & 3) * 16; // this warp's 16 x 16 piece
  const int items = tiles * nchunks;
  const bool vec = (ld & 1) == 0 && aligned16(Z) && (W == nullptr || aligned16(W));
  for (int it = tm.cta_rank(); it < items; it += ncta) {
    const int tile = it % tiles, ch = it / tiles;
    int ti, tj;
    if (SYM) {
      tj = 0;
      while ((tj + 1) * (tj + 2) / 2 <= tile)
        tj++;
      ti = tile - tj * (tj + 1) / 2; // ti <= tj
    } else {
      ti = tile % tp;
      tj = tile / tp;
    }
    const bool diag = SYM && ti == tj; // the B panel is the A panel
    const int64_t kb0 = (int64_t)ch * kb_per, kb1 = imin64(kb0 + kb_per, kblocks);
    // panel of 64 columns of X from column c0 (cols in all), rows 32 kb ..
    auto panel = [&](double *dst, const double *X, int c0, int cols, int64_t kb) {
      const int64_t r0 = kb * KR_GP;
      if (vec) {
#pragma unroll
        for (int e = threadIdx.x; e < KR_GT * KR_GP / 2; e += 512) {
          const int c = e / (KR_GP / 2), k = 2 * (e % (KR_GP / 2));
          const int64_t left = n - (r0 + k);
          const int live = c0 + c < cols && left > 0 ? (left > 1 ? 2 : 1) : 0;
          cp_async_f64<2>(dst + c * KR_GL + k, live ? X + (int64_t)(c0 + c) * ld + r0 + k : X, live);
        }
      } else {
#pragma unroll
        for (int e = threadIdx.x; e < KR_GT * KR_GP; e += 512) {
          const int c = e / KR_GP, k = e % KR_GP;
          const int live = c0 + c < cols && r0 + k < n;
          cp_async_f64<1>(dst + c * KR_GL + k, live ? X + (int64_t)(c0 + c) * ld + r0 + k : X, live);
        }
      }
    };
    auto stage = [&](int64_t kb) {
      if (kb < kb1) {
        double *st = kr_gemm_smem + (kb - kb0) % KR_GS * STAGE;
        panel(st, Z, ti * KR_GT, p, kb);
        if (SYM) {
          if (!diag)
            panel(st + PANEL, Z, tj * KR_GT, p, kb);
          if (two)
            panel(st + 2 * PANEL, W, tj * KR_GT, p, kb);
        } else {
          panel(st + PANEL, W, tj * KR_GT, q, kb);
        }
      }
      cp_async_commit();
    };
    // this warp's piece holds an element that is wanted
    const bool mine = ti * KR_GT + wr < p && tj * KR_GT + wc < (SYM ? p : q) && (!diag || wr <= wc);
    double aS[2][2][2], aG[2][2][2];
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int y = 0; y < 2; y++)
        aS[x][y][0] = aS[x][y][1] = aG[x][y][0] = aG[x][y][1] = 0.0;
#pragma unroll
    for (int s = 0; s < KR_GS - 1; s++)
      stage(kb0 + s);
    for (int64_t kb = kb0; kb < kb1; kb++) {
      cp_async_wait<KR_GS - 2>();
      __syncthreads(); // panel kb is there, and every warp has read panel kb - 1
      stage(kb + KR_GS - 1);
      if (mine) {
        const double *st = kr_gemm_smem + (kb - kb0) % KR_GS * STAGE;
        const double *fA = st + (wr + (lane >> 2)) * KR_GL + (lane & 3);
        const double *fB = st + (diag ? 0 : PANEL) + (wc + (lane >> 2)) * KR_GL + (lane & 3);
        const double *fC = st + 2 * PANEL + (wc + (lane >> 2)) * KR_GL + (lane & 3);
#pragma unroll
        for (int kk = 0; kk < KR_GP; kk += 4) {
          const double a0 = fA[kk], a1 = fA[kk + 8 * KR_GL];
          const double b0 = fB[kk], b1 = fB[kk + 8 * KR_GL];
          dmma_8x8x4(aS[0][0][0], aS[0][0][1], a0, b0);
          dmma_8x8x4(aS[0][1][0], aS[0][1][1], a0, b1);
          dmma_8x8x4(aS[1][0][0], aS[1][0][1], a1, b0);
          dmma_8x8x4(aS[1][1][0], aS[1][1][1], a1, b1);
          if (two) {
            const double c0 = fC[kk], c1 = fC[kk + 8 * KR_GL];
            dmma_8x8x4(aG[0][0][0], aG[0][0][1], a0, c0);
            dmma_8x8x4(aG[0][1][0], aG[0][1][1], a0, c1);
            dmma_8x8x4(aG[1][0][0], aG[1][0][1], a1, c0);
            dmma_8x8x4(aG[1][1][0], aG[1][1][1], a1, c1);
          }
        }
      }
    }
    cp_async_wait<0>();
    __syncthreads(); // the next item's panels may be staged
    if (mine) {
      double *pt = part + (size_t)it * ITEM;
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int y = 0; y < 2; y++) {
          const int i = wr + 8 * x + (lane >> 2), j = wc + 8 * y + 2 * (lane & 3);
          pt[i + j * KR_GT] = aS[x][y][0];
          pt[i + (j + 1) * KR_GT] = aS[x][y][1];
          if (two) {
            pt[KR_GT * KR_GT + i + j * KR_GT] = aG[x][y][0];
            pt[KR_GT * KR_GT + i + (j + 1) * KR_GT] = aG[x][y][1];
          }
        }
    }
  }
  tm.sync();
  const int64_t nthr = tm.nthreads();
  for (int64_t e = tm.tid(); e < (int64_t)p * q; e += nthr) {
    const int i = (int)(e % p), j = (int)(e / p);
    if (SYM && i > j)
      continue;
    const int ti = i / KR_GT, tj = j / KR_GT, li = i % KR_GT, lj = j % KR_GT;
    const int tile = SYM ? tj * (tj + 1) / 2 + ti : tj * tp + ti;
    double sv = 0.0, gv = 0.0;
    for (int ch = 0; ch < nchunks; ch++) {
      const double *pt = part + (size_t)(tile + ch * tiles) * ITEM;
      sv += __ldcg(pt + li + lj * KR_GT);
      if (two)
        gv += __ldcg(pt + KR_GT * KR_GT + li + lj * KR_GT);
    }
    S[i + (size_t)j * p] = sv;
    if (SYM) {
      S[j + (size_t)i * p] = sv;
      if (two) {
        G[i + (size_t)j * p] = gv;
        G[j + (size_t)i * p] = gv;
      }
    }
  }
  tm.sync();
}

// C = A^T B: the tiled kernel for long products with wide blocks, where the
// shared-memory panels pay off; the direct one (one warp per 8 x 8 tile,
// operands straight from global memory) for short or narrow ones, where
// streaming full 64-column panels 16 rows at a time through one block costs
// more than it saves (measured: a 1000-row LOBPCG with 3-column blocks ran
// 3.3x slower tiled). `part` must suit both (see each).
template <class Team>
KR_DEV void team_gemm_tn(Team &tm, int64_t n, const double *A, int a, const double *B, int b, int64_t ld,
                         double *C, double *part) {
  if (n >= KR_TN_ROWS && (a >= KR_TN_COLS || b >= KR_TN_COLS))
    team_tn_panels<false>(tm, n, A, a, B, b, ld, C, nullptr, part);
  else
    team_tn_direct<false>(tm, n, A, a, B, b, ld, C, nullptr, part);
}

// ---- Z * Y products (combine_columns, LOBPCGSolver.cpp:122-134) -----------
// out (n x q) = Z (n x zc) * Y[roff : roff + zc, 0 : q], or out -= that
// product; Z and out column-major with leading dim ld, Y column-major with
// leading dim ldy. On the FP64 tensor cores: a block takes 64-row tiles of
// the tall operand (every 128-column group of the output for one tile before
// the next tile, so the tile is read from HBM once); k runs in chunks of 16
// staged in shared memory, the next on its way by cp.async across the ends of
// tiles; each of the 16 warps owns a 16 x 32 piece of the 64 x 128 output
// group (2 x 4 DMMA 8x8 tiles), dealt so that pieces past the last column fall
// to the SM's four pipes alike. Each output is summed in a fixed order,
// independent of the team. Bound by the DMMA pipe; both chunk pitches put a
// fragment on distinct banks (4194304 x 288 times 288 x 96: 15.1 -> 25.8
// TFLOP/s). Needs 512 threads and gemm_nn_smem_bytes() of dynamic shared memory.
#define KR_NT 64  // rows per tile
#define KR_NQ 128 // output columns per group
#define KR_NK 16  // k per chunk
#define KR_NZL (KR_NT + 4) // pitch of a k row of the Z chunk
#define KR_NYL (KR_NK + 4) // pitch of a column of the Y chunk
#define KR_NS 2            // chunks held: one multiplied, one on its way
__host__ __device__ constexpr size_t gemm_nn_smem_bytes() {
  return (size_t)KR_NS * (KR_NK * KR_NZL + KR_NQ * KR_NYL) * 8;
}

// Narrow form (q <= KR_NQ_DIRECT outputs): every thread takes whole rows and
// sums over k in order on the CUDA cores, with no shared memory and no
// barrier. For the few-column blocks of small solves the tiled form spends
// two block barriers per 64-row tile on a 64 x 128 output group it barely
// fills; this form costs none (the caller's barrier publishes the result). Bound
// by the latency of a row's loads: those of U = 8 k are issued together in the
// kernel of its own (36 x 12 at n = 20011: 33.9 -> 18.5 us, at n = 1000003 221 ->
// 183), one k at a time inside the solver, whose registers are short (eight: 3%
// slower solves at 4 and 6 columns, 3% faster at 16).
#define KR_NQ_DIRECT 16
template <int U, class Team>
KR_DEV void team_gemm_nn_direct(Team &tm, int64_t n, const double *Z, int64_t ld, int zc, const double *Y, int ldy,
                                int roff, int q, double *out, bool subtract) {
  for (int64_t i = tm.tid(); i < n; i += tm.nthreads()) {
    double acc[KR_NQ_DIRECT];
#pragma unroll
    for (int j = 0; j < KR_NQ_DIRECT; j++)
      acc[j] = 0.0;
    int k = 0;
    for (; k + U <= zc; k += U) {
      double z[U];
#pragma unroll
      for (int u = 0; u < U; u++)
        z[u] = Z[(int64_t)(k + u) * ld + i];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const double *yk = Y + roff + k + u;
#pragma unroll
        for (int j = 0; j < KR_NQ_DIRECT; j++)
          if (j < q)
            acc[j] += z[u] * yk[(int64_t)j * ldy];
      }
    }
    for (; k < zc; k++) {
      const double z = Z[(int64_t)k * ld + i];
      const double *yk = Y + roff + k;
#pragma unroll
      for (int j = 0; j < KR_NQ_DIRECT; j++)
        if (j < q)
          acc[j] += z * yk[(int64_t)j * ldy];
    }
#pragma unroll
    for (int j = 0; j < KR_NQ_DIRECT; j++)
      if (j < q) {
        double *o = out + (int64_t)j * ld + i;
        *o = subtract ? *o - acc[j] : acc[j];
      }
  }
}

template <class Team>
KR_DEV void team_gemm_nn(Team &tm, int64_t n, const double *Z, int64_t ld, int zc, const double *Y, int ldy,
                         int roff, int q, double *out, bool subtract) {
  if (q <= KR_NQ_DIRECT) {
    team_gemm_nn_direct<1>(tm, n, Z, ld, zc, Y, ldy, roff, q, out, subtract);
    return;
  }
  extern __shared__ __align__(16) double kr_gemm_smem[];
  constexpr int STAGE = KR_NK * KR_NZL + KR_NQ * KR_NYL;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int wr = (wid >> 2) * 16, wc = ((wid + (wid >> 2)) & 3) * 32; // this warp's 16 x 32 piece
  const int64_t row_tiles = (n + KR_NT - 1) / KR_NT;
  const int col_groups = (q + KR_NQ - 1) / KR_NQ;
  const int nchunks = (zc + KR_NK - 1) / KR_NK;
  const bool vz = (ld & 1) == 0 && aligned16(Z);
  const bool vy = ((ldy | roff) & 1) == 0 && aligned16(Y);
  const int64_t ncta = tm.ncta(), rt0 = tm.cta_rank();
  if (rt0 >= row_tiles)
    return;
  // steps of this block: (row tile, column group, chunk), chunk fastest
  struct Step {
    int64_t rt;
    int cg, ch;
  };
  auto next = [&](Step &s) {
    if (++s.ch == nchunks) {
      s.ch = 0;
      if (++s.cg == col_groups) {
        s.cg = 0;
        s.rt += ncta;
      }
    }
  };
  auto stage = [&](const Step &s, int slot) {
    if (s.rt < row_tiles) {
      double *sZ = kr_gemm_smem + slot * STAGE, *sY = sZ + KR_NK * KR_NZL;
      const int64_t r0 = s.rt * KR_NT;
      const int c0 = s.cg * KR_NQ, k0 = s.ch * KR_NK;
      if (vz) {
        const int kk = threadIdx.x / (KR_NT / 2), r = 2 * (threadIdx.x % (KR_NT / 2)); // 512 pairs
        const int64_t left = n - (r0 + r);
        const int live = k0 + kk < zc && left > 0 ? (left > 1 ? 2 : 1) : 0;
        cp_async_f64<2>(sZ + kk * KR_NZL + r, live ? Z + (int64_t)(k0 + kk) * ld + r0 + r : Z, live);
      } else {
#pragma unroll
        for (int e = threadIdx.x; e < KR_NT * KR_NK; e += 512) {
          const int kk = e / KR_NT, r = e % KR_NT;
          const int live = k0 + kk < zc && r0 + r < n;
          cp_async_f64<1>(sZ + kk * KR_NZL + r, live ? Z + (int64_t)(k0 + kk) * ld + r0 + r : Z, live);
        }
      }
      if (vy) {
#pragma unroll
        for (int e = threadIdx.x; e < KR_NQ * KR_NK / 2; e += 512) {
          const int c = e / (KR_NK / 2), kk = 2 * (e % (KR_NK / 2));
          const int left = zc - (k0 + kk);
          const int live = c0 + c < q && left > 0 ? (left > 1 ? 2 : 1) : 0;
          cp_async_f64<2>(sY + c * KR_NYL + kk, live ? Y + (int64_t)(roff + k0 + kk) + (int64_t)(c0 + c) * ldy : Y,
                          live);
        }
      } else {
#pragma unroll
        for (int e = threadIdx.x; e < KR_NQ * KR_NK; e += 512) {
          const int c = e / KR_NK, kk = e % KR_NK;
          const int live = c0 + c < q && k0 + kk < zc;
          cp_async_f64<1>(sY + c * KR_NYL + kk, live ? Y + (int64_t)(roff + k0 + kk) + (int64_t)(c0 + c) * ldy : Y,
                          live);
        }
      }
    }
    cp_async_commit();
  };
  Step ahead{rt0, 0, 0};
  for (int s = 0; s < KR_NS - 1; s++) {
    stage(ahead, s);
    next(ahead);
  }
  double acc[2][4][2];
  int slot = 0;
  for (Step now{rt0, 0, 0}; now.rt < row_tiles; next(now)) {
    cp_async_wait<KR_NS - 2>();
    __syncthreads(); // this chunk is there, and every warp has read the one before
    stage(ahead, (slot + KR_NS - 1) % KR_NS);
    next(ahead);
    if (now.ch == 0) {
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int y = 0; y < 4; y++)
          acc[x][y][0] = acc[x][y][1] = 0.0;
    }
    const int c0 = now.cg * KR_NQ;
    if (c0 + wc < q) { // warp-uniform: warps past the last column have nothing to do
      const double *sZ = kr_gemm_smem + slot * STAGE, *sY = sZ + KR_NK * KR_NZL;
      const double *fA = sZ + (lane & 3) * KR_NZL + wr + (lane >> 2);
      const double *fB = sY + (wc + (lane >> 2)) * KR_NYL + (lane & 3);
#pragma unroll
      for (int kk = 0; kk < KR_NK; kk += 4) {
        double fa[2], fb[4];
#pragma unroll
        for (int x = 0; x < 2; x++)
          fa[x] = fA[kk * KR_NZL + 8 * x];
#pragma unroll
        for (int y = 0; y < 4; y++)
          fb[y] = fB[8 * y * KR_NYL + kk];
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
          for (int y = 0; y < 4; y++)
            dmma_8x8x4(acc[x][y][0], acc[x][y][1], fa[x], fb[y]);
      }
      if (now.ch == nchunks - 1) {
        const int64_t r0 = now.rt * KR_NT;
#pragma unroll
        for (int x = 0; x < 2; x++)
#pragma unroll
          for (int y = 0; y < 4; y++) {
            const int64_t i = r0 + wr + 8 * x + (lane >> 2);
            const int j = c0 + wc + 8 * y + 2 * (lane & 3);
            if (i < n) {
#pragma unroll
              for (int h = 0; h < 2; h++)
                if (j + h < q) {
                  double *o = out + (int64_t)(j + h) * ld + i;
                  *o = subtract ? *o - acc[x][y][h] : acc[x][y][h];
                }
            }
          }
      }
    }
    slot = (slot + 1) % KR_NS;
  }
  cp_async_wait<0>();
  __syncthreads(); // the next product may stage its chunks
}

// X[:, i] -= sum_j S[:, j] * Cc(j, i) for i < k, j < ns (X, S column-major
// with leading dim ld; Cc leading dim ldc).
template <class Team>
KR_DEV void team_combine_sub(Team &tm, int64_t n, const double *S, int64_t ld, int ns, const double *Cc, int ldc,
                             int k, double *X) {
  team_gemm_nn(tm, n, S, ld, ns, Cc, ldc, 0, k, X, true);
}

// out[:, i] = sum_j Y(roff + j, i) * Z[:, j], i < q, j < zc (column-major,
// both with leading dim ld; Y leading dim ldy).
template <class Team>
KR_DEV void team_combine(Team &tm, int64_t n, const double *Z, int64_t ld, int zc, const double *Y,
                         int ldy, int roff, int q, double *out) {
  team_gemm_nn(tm, n, Z, ld, zc, Y, ldy, roff, q, out, false);
}

} // namespace kr
