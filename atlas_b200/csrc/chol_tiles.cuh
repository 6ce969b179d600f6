// Cholesky factorization (FP64, order <= 256) by one CTA, left-looking over
// 16-column panels kept as 16 x 16 tiles in shared memory.  Used by the
// batched solver (batched.cu) for whole problems and by potrf (chol.cu) for
// its diagonal blocks.
//
// What bounds it: the chain of columns in the diagonal tiles (1/sqrt, the
// multipliers, the next diagonal entry: about 150 cycles a column), not
// bandwidth or the FP64 pipes.  So one warp owns that chain, factoring the
// diagonal tile in registers by shuffles, and everything else runs beside it:
//   * phase 1 of panel j: warp 0 adds panel j-1's product to diagonal tile j
//     and factors it; the other warps add the same product to the rest of
//     panel j and all earlier panels' products to panel j+1 (FP64 tensor
//     cores, accumulators started from the tile), while the copies of panel
//     j+2 from global memory are in flight;
//   * phase 2: every thread solves one row of the panel against the diagonal
//     tile and writes it out.  Two barriers per panel.
// Left-looking, because a finished row of tiles is dead as soon as its own
// panel is done: at most 79 of the 136 tiles of order 256 are live at once
// (162 KB), so A crosses global memory once each way and never returns.
//
// Right-hand sides: up to eight ride along as one extra block row (B^T), so
// the forward substitution is part of the factorization.
#pragma once
#include <cuda_runtime.h>
#include "common.cuh"
#include "chol_blocks.cuh"

namespace atlb {
namespace cholt {

constexpr int TB = 16;          // tile order
constexpr int MAXNB = 16;       // tiles per side (order 256)
constexpr int TILE = TB * TB;   // doubles per tile
constexpr int RHS = 8;          // right-hand sides per block row
constexpr int RTILE = RHS * TB;

// Where tile (i, k) of a matrix of nb tiles a side lives in the pool, and how
// many tiles the pool needs.  Panels j+1 and j+2 get their places before
// panel j+1 is worked on; block row j's places are free once panel j is done.
struct SlotTable {
  unsigned char slot[MAXNB + 1][MAXNB][MAXNB];
  unsigned char need[MAXNB + 1];
};
constexpr SlotTable make_slots() {
  SlotTable t{};
  for (int nb = 1; nb <= MAXNB; nb++) {
    unsigned char free_list[MAXNB * MAXNB] = {};
    int nfree = 0, top = 0;
    for (int c = 0; c < nb; c++) {
      // panel c is placed in phase 1 of panel c - 2, when the rows up to c - 3 are free
      if (c >= 3)
        for (int k = 0; k <= c - 3; k++) free_list[nfree++] = t.slot[nb][c - 3][k];
      for (int i = c; i < nb; i++) {
        if (nfree > 0) t.slot[nb][i][c] = free_list[--nfree];
        else t.slot[nb][i][c] = (unsigned char)top++;
      }
    }
    t.need[nb] = (unsigned char)top;
  }
  return t;
}
constexpr SlotTable kSlotsHost = make_slots();
static __constant__ SlotTable kSlots = make_slots();

// Tiles the pool holds for nb tiles a side: the factorization's own, and at
// least two panels plus the right-hand sides' rows for the streamed solves.
constexpr int pool_tiles(int nb, bool solve) {
  const int f = kSlotsHost.need[nb], s = solve ? 2 * nb + (nb + 1) / 2 : 0;
  return f > s ? f : s;
}
constexpr int pool_tiles_upto(int nb, bool solve) {
  int m = 0;
  for (int b = 1; b <= nb; b++) m = pool_tiles(b, solve) > m ? pool_tiles(b, solve) : m;
  return m;
}

// Element (r, c) of a tile: column-major with the row's bits 2-3 exchanged by
// the column's low bits, so that the 8 x 4 operand fragments of the FP64 MMA
// (16 lanes: 4 rows x 4 columns) and a column's 16 rows fall in distinct
// banks.  The right-hand sides' tiles (8 rows) do the same with bit 2.
__device__ __forceinline__ int at(int r, int c) { return c * TB + (r ^ ((c & 3) << 2)); }
__device__ __forceinline__ int rat(int r, int c) { return c * RHS + (r ^ ((c & 2) << 1)); }

template <int NB>  // up to NB tiles a side
struct Shared {
  double D[TILE];       // the current diagonal tile of L, D[c * 16 + k] = L(k, c)
  double rinv[TB * NB]; // 1 / L(c, c)
  double t[RHS * TB];
  unsigned char slot[NB][MAXNB];  // kSlots of this order
  int fail, stored;
};

// The operand fragments of one 16-column tile pair: a = rows of -L_i, b = rows of L_j.
struct Frags {
  double a[4][2], b[4][2];
};
__device__ __forceinline__ void load_frags(Frags &f, const double *Li, const double *Lj) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      f.a[q][h] = Li[at(g + 8 * h, 4 * q + t)];
      f.b[q][h] = Lj[at(g + 8 * h, 4 * q + t)];
    }
}
__device__ __forceinline__ void mma_tile(double (&acc)[2][2][2], const Frags &f) {
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
      for (int h = 0; h < 2; h++) cholb::dmma_8x8x4(acc[a][h], -f.a[q][a], f.b[q][h]);
}

// tile(i, c) -= sum over k in [k0, k1) of L(i, k) L(c, k)^T by one warp; four
// accumulators, because a dependent FP64 MMA waits 26 cycles for the one
// before, and the next tile pair's fragments are loaded under the products
__device__ __forceinline__ void update_tile(double *pool, const unsigned char (*sl)[MAXNB], int i, int c, int k0,
                                            int k1) {
  if (k0 >= k1) return;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double *C = pool + (int)sl[i][c] * TILE;
  double acc[2][2][2];
  Frags f;
  load_frags(f, pool + (int)sl[i][k0] * TILE, pool + (int)sl[c][k0] * TILE);
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) acc[a][h][e] = C[at(g + 8 * a, 8 * h + 2 * t + e)];
#pragma unroll 1
  for (int k = k0 + 1; k < k1; k++) {
    Frags nx;
    load_frags(nx, pool + (int)sl[i][k] * TILE, pool + (int)sl[c][k] * TILE);
    mma_tile(acc, f);
    f = nx;
  }
  mma_tile(acc, f);
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) C[at(g + 8 * a, 8 * h + 2 * t + e)] = acc[a][h][e];
}
// the same for the right-hand sides' rows
__device__ __forceinline__ void update_rhs(double *pool, const unsigned char (*sl)[MAXNB], double *rhs, int c, int k0,
                                           int k1) {
  if (k0 >= k1) return;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double *C = rhs + c * RTILE;
  double acc[2][2];
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int e = 0; e < 2; e++) acc[h][e] = C[rat(g, 8 * h + 2 * t + e)];
#pragma unroll 1
  for (int k = k0; k < k1; k++) {
    const double *Lr = rhs + k * RTILE, *Lj = pool + (int)sl[c][k] * TILE;
    double a[4], b[4][2];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      a[q] = Lr[rat(g, 4 * q + t)];
      b[q][0] = Lj[at(g, 4 * q + t)];
      b[q][1] = Lj[at(g + 8, 4 * q + t)];
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int h = 0; h < 2; h++) cholb::dmma_8x8x4(acc[h], -a[q], b[q][h]);
  }
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int e = 0; e < 2; e++) C[rat(g, 8 * h + 2 * t + e)] = acc[h][e];
}

// Factor the jb <= 16 columns of diagonal tile T (one warp; lane i and lane
// i + 16 hold row i).  Every lane carries its own diagonal entry, so the
// chain from column to column is: the diagonal by shuffle, 1/sqrt, this
// lane's multiplier, its next diagonal entry; the other lanes' multipliers
// come back from D two at a time (shuffling them doubled the instructions).  L(k, c) goes to D[c * 16 + k],
// 1/L(c, c) to rinv; columns from the first non-positive pivot on are not
// stored.  Returns 0 or that pivot's 1-based column.
__device__ __forceinline__ int factor_diag(const double *T, int jb, double *D, double *rinv) {
  const int lane = threadIdx.x & 31, i = lane & 15;
  double r[TB];
#pragma unroll
  for (int k = 0; k < TB; k++) r[k] = T[at(i, k)];
  double dg = i < jb ? T[at(i, i)] : 1.0;
  int fail = 0;
  double d = __shfl_sync(0xffffffffu, dg, 0);
#pragma unroll
  for (int c = 0; c < TB; c++) {
    if (!(d > 0.0) && !fail) fail = c + 1;  // later columns run on, unused
    const double ri = rsqrt(d), l = (i == c ? d : r[c]) * ri;
    dg = fma(-l, l, dg);
    if (c + 1 < TB) d = __shfl_sync(0xffffffffu, dg, c + 1);
    if (lane < TB) D[c * TB + i] = l;  // above the diagonal: not a value anyone reads
    if (lane == 0) rinv[c] = ri;
    __syncwarp();
#pragma unroll
    for (int k = (c + 1) & ~1; k < TB; k += 2) {
      const double2 m = *reinterpret_cast<const double2 *>(D + c * TB + k);
      if (k > c) r[k] = fma(-l, m.x, r[k]);
      r[k + 1] = fma(-l, m.y, r[k + 1]);
    }
  }
  return fail;
}

// Factor the n x n (1 <= n <= 256) matrix at A: lower triangle column-major
// (UP: the upper triangle, factored as the transpose of the lower one), and
// apply the forward substitution to the first nr <= 8 columns of B (left in
// rhs, rhs tile k holding entries 16k..16k+15).  pool: pool_tiles(nb) tiles;
// rhs: nb tiles of 8 x 16.  Returns 0 or the first non-positive pivot
// (1-based), the same in every thread; A then holds the factor's columns
// before that pivot's panel (and, within the diagonal tile, before the
// pivot), the rest of A unchanged.
template <int NT, bool UP, int NB>
__device__ int factor(int n, double *A, long lda, const double *B, long ldb, int nr, double *pool, double *rhs,
                      Shared<NB> &S) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int NW = NT / 32, NC = NT - 32;  // warps 1.. copy panels in
  const int nb = (n + TB - 1) / TB;
  const unsigned char(*sl)[MAXNB] = S.slot;
  for (int idx = tid; idx < nb * MAXNB; idx += NT) S.slot[0][idx] = kSlots.slot[nb][0][idx];
  __syncthreads();
  // panel c of A (and of B^T) into its tiles, zero beyond the matrix
  auto load_panel = [&](int c, int id, int step) {
    const int tot = (nb - c) * TILE;
#pragma unroll 2
    for (int idx = id; idx < tot; idx += step) {
      const int i = c + (idx >> 8);
      const int r = UP ? (idx >> 4) & 15 : idx & 15, q = UP ? idx & 15 : (idx >> 4) & 15;
      const int gi = i * TB + r, gk = c * TB + q;
      const bool p = gi < n && gk < n && (i > c || r >= q);
      const double *g = UP ? A + gk + (long)gi * lda : A + gi + (long)gk * lda;
      cp_async8(pool + (int)sl[i][c] * TILE + at(r, q), p ? g : A, p);
    }
    if (nr > 0)
      for (int idx = id; idx < RTILE; idx += step) {
        const int q = idx & 15, r = idx >> 4, gk = c * TB + q;
        const bool p = r < nr && gk < n;
        cp_async8(rhs + c * RTILE + rat(r, q), p ? B + gk + (long)r * ldb : A, p);
      }
  };
  if (tid == 0) S.fail = 0;
#pragma unroll 1
  for (int c = 0; c < min(nb, 2); c++) load_panel(c, tid, NT);
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
#pragma unroll 1
  for (int j = 0; j < nb; j++) {
    const int jb = min(TB, n - j * TB);
    // phase 1
    if (warp == 0) {
      update_tile(pool, sl, j, j, max(0, j - 1), j);
      __syncwarp();
      const int f = factor_diag(pool + (int)sl[j][j] * TILE, jb, S.D, S.rinv + j * TB);
      if (lane == 0) {
        S.stored = f ? f - 1 : jb;
        if (f) S.fail = j * TB + f;
      }
      if (jb < TB)  // columns the matrix does not have solve to zero
        for (int idx = jb * TB + lane; idx < TILE; idx += 32) {
          S.D[idx] = 0.0;
          S.rinv[j * TB + (idx >> 4)] = 0.0;
        }
    } else {
      if (j + 2 < nb) load_panel(j + 2, tid - 32, NC);
#pragma unroll 1
      for (int i = j + warp; i <= nb; i += NW - 1)
#pragma unroll 1
        for (int c = j; c <= min(j + 1, nb - 1); c++) {
          const int k0 = c == j ? max(0, j - 1) : 0;
          if (i < nb) update_tile(pool, sl, i, c, k0, j);
          else if (nr > 0) update_rhs(pool, sl, rhs, c, k0, j);
        }
    }
    __syncthreads();
#pragma unroll 1
    for (int idx = tid; idx < TILE; idx += NT) {  // the diagonal tile goes out
      const int c = idx >> 4, i = idx & 15;
      if (i >= c && i < jb && c < S.stored) {
        if (UP) A[j * TB + c + (long)(j * TB + i) * lda] = S.D[idx];
        else A[j * TB + i + (long)(j * TB + c) * lda] = S.D[idx];
      }
    }
    if (S.fail) break;
    // phase 2: rows below the diagonal tile, and the right-hand sides
    const int nrow = (nb - 1 - j) * TB;
#pragma unroll 1
    for (int row = tid; row < nrow + nr; row += NT) {
      const bool isr = row >= nrow;
      const int i = j + 1 + (row >> 4), rr = isr ? row - nrow : row & 15;
      double *T = isr ? rhs + j * RTILE : pool + (int)sl[i][j] * TILE;
      double x[TB];
#pragma unroll
      for (int c = 0; c < TB; c++) x[c] = T[isr ? rat(rr, c) : at(rr, c)];
#pragma unroll
      for (int c = 0; c < TB; c++) {
        x[c] *= S.rinv[j * TB + c];
#pragma unroll
        for (int k = (c + 1) & ~1; k < TB; k += 2) {
          const double2 d = *reinterpret_cast<const double2 *>(S.D + c * TB + k);
          if (k > c) x[k] = fma(-x[c], d.x, x[k]);
          x[k + 1] = fma(-x[c], d.y, x[k + 1]);
        }
      }
#pragma unroll
      for (int c = 0; c < TB; c++) T[isr ? rat(rr, c) : at(rr, c)] = x[c];
      const int gi = i * TB + rr;
      if (!isr && gi < n) {  // a panel with rows below it is 16 columns wide
#pragma unroll
        for (int c = 0; c < TB; c++) {
          if (UP) A[j * TB + c + (long)gi * lda] = x[c];
          else A[gi + (long)(j * TB + c) * lda] = x[c];
        }
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  }
  cp_async_commit();  // after a failure, copies of a later panel may be on their way
  cp_async_wait<0>();
  __syncthreads();
  const int fail = S.fail;
  __syncthreads();
  return fail;
}

// One pass of substitutions with L (n x n lower, global memory, its diagonal's
// reciprocals in S.rinv) over nr <= 8 right-hand sides held in xs
// (xs[r * 16 nb + i]): backward solves L^T x = y (panels from the last to
// the first), otherwise L y = b.  L's panels stream through two buffers of
// nb tiles each (cp.async, one panel ahead); tile element (rr, c) sits at
// c * 16 + (rr ^ c), conflict-free by rows and by columns.
template <int NT, bool backward, int NB>
__device__ void stream_solve(int n, const double *A, long lda, int nr, double *xs, double *ring,
                             Shared<NB> &S) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int NW = NT / 32;
  const int nb = (n + TB - 1) / TB, np = nb * TB;
  auto fetch = [&](int s) {
    if (s < nb) {
      const int j = backward ? nb - 1 - s : s;
      double *P = ring + (s & 1) * nb * TILE;
      const int tot = (nb - j) * TILE;
#pragma unroll 2
      for (int idx = tid; idx < tot; idx += NT) {
        const int i = j + (idx >> 8), r = idx & 15, q = (idx >> 4) & 15;
        const int gi = i * TB + r, gk = j * TB + q;
        const bool p = gi < n && gk < n && (i > j || r >= q);
        cp_async8(P + (idx & ~255) + q * TB + (r ^ q), p ? A + gi + (long)gk * lda : A, p);
      }
    }
    cp_async_commit();
  };
  fetch(0);
#pragma unroll 1
  for (int s = 0; s < nb; s++) {
    const int j = backward ? nb - 1 - s : s;
    fetch(s + 1);
    cp_async_wait<1>();
    __syncthreads();
    const double *P = ring + (s & 1) * nb * TILE;
    if (backward) {  // t(c) = sum over the rows below of L(i, c) x(i): half a warp per column
      const int rr = tid & 15;
#pragma unroll 1
      for (int c = tid >> 4; c < TB; c += NT / 16) {
        double acc[RHS];
#pragma unroll
        for (int r = 0; r < RHS; r++) acc[r] = 0.0;
#pragma unroll 2
        for (int i = 1; i < nb - j; i++) {
          const double l = P[i * TILE + c * TB + (rr ^ c)];
          const double *x = xs + (j + i) * TB + rr;
#pragma unroll
          for (int r = 0; r < RHS; r++)
            if (r < nr) acc[r] = fma(l, x[r * np], acc[r]);
        }
#pragma unroll
        for (int r = 0; r < RHS; r++)
          if (r < nr) {
#pragma unroll
            for (int o = 8; o; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
            if (rr == 0) S.t[r * TB + c] = acc[r];
          }
      }
      __syncthreads();
    }
#pragma unroll 1
    for (int r = warp; r < nr; r += NW) {  // the diagonal tile: one warp per right-hand side
      const int c = lane & 15;
      double v = xs[r * np + j * TB + c];
      double l[TB];
      if (backward) {
        v -= S.t[r * TB + c];
#pragma unroll
        for (int q = 0; q < TB; q++) l[q] = q > c ? P[c * TB + (q ^ c)] : 0.0;  // L(q, c)
      } else {
#pragma unroll
        for (int q = 0; q < TB; q++) l[q] = q < c ? P[q * TB + (c ^ q)] : 0.0;  // L(c, q)
      }
      const double ri = S.rinv[j * TB + c];
#pragma unroll
      for (int u = 0; u < TB; u++) {
        const int q = backward ? TB - 1 - u : u;
        if (c == q) v *= ri;
        const double xq = __shfl_sync(0xffffffffu, v, q);
        v = fma(-l[q], xq, v);
      }
      if (lane < TB) xs[r * np + j * TB + c] = v;
    }
    __syncthreads();
    if (!backward) {
#pragma unroll 1
      for (int row = tid; row < (nb - 1 - j) * TB; row += NT) {
        const int i = 1 + (row >> 4), rr = row & 15;
        double l[TB];
#pragma unroll
        for (int c = 0; c < TB; c++) l[c] = P[i * TILE + c * TB + (rr ^ c)];
#pragma unroll
        for (int r = 0; r < RHS; r++)
          if (r < nr) {
            double acc = xs[r * np + (j + i) * TB + rr];
#pragma unroll
            for (int c = 0; c < TB; c++) acc = fma(-l[c], xs[r * np + j * TB + c], acc);
            xs[r * np + (j + i) * TB + rr] = acc;
          }
      }
      __syncthreads();
    }
  }
  cp_async_wait<0>();
  __syncthreads();
}

// L L^T X = B for all nrhs columns of B after factor(): the first eight
// columns' forward substitution is in rhs already.  Uses the pool as
// workspace (pool_tiles(nb, true) tiles).
template <int NT, int NB>
__device__ void solve(int n, const double *A, long lda, double *B, long ldb, int nrhs, double *pool,
                      const double *rhs, Shared<NB> &S) {
  const int tid = threadIdx.x, nb = (n + TB - 1) / TB, np = nb * TB;
  double *xs = pool, *ring = pool + (nb + 1) / 2 * TILE;  // 8 x 16 nb values take nb / 2 tiles
#pragma unroll 1
  for (int r0 = 0; r0 < nrhs; r0 += RHS) {
    const int nr = min(RHS, nrhs - r0);
    double *Bc = B + (long)r0 * ldb;
#pragma unroll 1
    for (int idx = tid; idx < nr * np; idx += NT) {
      const int r = idx / np, i = idx - r * np;
      xs[idx] = r0 == 0 ? rhs[(i >> 4) * RTILE + rat(r, i & 15)] : (i < n ? Bc[i + (long)r * ldb] : 0.0);
    }
    __syncthreads();
    if (r0 > 0) stream_solve<NT, false>(n, A, lda, nr, xs, ring, S);
    stream_solve<NT, true>(n, A, lda, nr, xs, ring, S);
#pragma unroll 1
    for (int idx = tid; idx < nr * np; idx += NT) {
      const int r = idx / np, i = idx - r * np;
      if (i < n) Bc[i + (long)r * ldb] = xs[idx];
    }
    __syncthreads();
  }
}

}  // namespace cholt
}  // namespace atlb
