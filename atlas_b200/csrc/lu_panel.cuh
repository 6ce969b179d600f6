// The LU panel of one CTA, one thread a row, and the update behind it (lu.cu's
// panels of few rows, the batched LU).
#pragma once
#include <cfloat>
#include <climits>
#include "chol_blocks.cuh"
#include "pivot.cuh"

namespace atlb {

constexpr int LPW = 16;          // panel width
constexpr int LU_LDU = LPW + 4;  // U12 copy, U(q, k) at k * LU_LDU + q

// The shared memory SM has: P[LPW * LDP], the panel (LDP = 4 mod 16: the MMA's
// fragments fall in distinct banks); U; per-warp candidate rows, their keys and
// positions by column parity, cand[2][NT / 32][LPW], ckey, cpos; piv[], the
// pivots; fail, the first zero pivot (1-based) or 0.

// a[]: this thread's row of the panel (row tid of m, jb <= 16
// columns); returns its final position.  The row is shifted as columns are
// finished -- a[0] is always the current column -- so the loop is one small
// body (unrolled, the sixteen bodies overflow the instruction cache);
// multipliers, and the U part of a pivot row, go to S.P at the thread's own
// row, from where the caller takes the finished row.  A column without a nonzero
// candidate takes the row at its position; with ZERO a zero goes before a NaN.
template <int NT, bool ZERO, class SM>
__device__ __forceinline__ int lu_panel(SM &S, double (&a)[LPW], int m, int jb, int j0) {
  constexpr int NW = NT / 32, LDP = SM::LDP;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool act = tid < m, chosen = false;
  int pos = tid;
#pragma unroll 1
  for (int c = 0; c < jb; c++) {
    const int b = c & 1;
    // without ZERO a zero or NaN entry never wins, except that the row at position
    // c stands in when there is no other candidate (then: no interchange)
    unsigned long long key = 0;
    if (act) key = ZERO || fabs(a[0]) > 0.0 ? pivot_key(a[0]) : (pos == c ? 1ull : 0ull);
    const int wl = warp_argmax_lane(key, act ? (unsigned)pos : 0xffffffffu);
    if (lane == wl) {
      S.ckey[b][warp] = key;
      S.cpos[b][warp] = act ? pos : INT_MAX;
#pragma unroll
      for (int k = 0; k < LPW; k += 2)
        *reinterpret_cast<double2 *>(&S.cand[b][warp][k]) = make_double2(a[k], a[k + 1]);
    }
    __syncthreads();
    int w = 0;
    if (NW > 1) w = warp_argmax_lane(lane < NW ? S.ckey[b][lane] : 0ull, lane < NW ? (unsigned)S.cpos[b][lane] : 0xffffffffu);
    const int p = S.cpos[b][w];
    const double *u = S.cand[b][w];
    const double piv = u[0];
    if (tid == 0) {
      S.piv[j0 + c] = j0 + p;
      if (piv == 0.0 && !S.fail) S.fail = j0 + c + 1;
    }
    if (act) {
      if (pos == p) {  // the pivot row: it keeps its place in a[] from here on
        act = false;
        chosen = true;
        pos = c;
      } else {
        if (pos == c) pos = p;
        const bool nz = piv != 0.0;  // a zero pivot leaves the column unscaled and the row unchanged
        const double l = !nz ? a[0] : fabs(piv) >= DBL_MIN ? a[0] * (1.0 / piv) : a[0] / piv;
        S.P[c * LDP + tid] = l;
        if (nz) {
#pragma unroll
          for (int k = 0; k < LPW; k += 2) {
            const double2 v = *reinterpret_cast<const double2 *>(u + k);
            if (k > 0) a[k - 1] = fma(-l, v.x, a[k]);
            a[k] = fma(-l, v.y, a[k + 1]);
          }
        } else {
#pragma unroll
          for (int k = 1; k < LPW; k++) a[k - 1] = a[k];
        }
        a[LPW - 1] = 0.0;
      }
    }
  }
  if (chosen) {
#pragma unroll
    for (int k = 0; k < LPW; k++)
      if (pos + k < jb) S.P[(pos + k) * LDP + tid] = a[k];
  }
  return pos;
}

// C (mt x nt, global, ldc) -= P (mt x 16, shared) U (16 x nt, shared); each warp
// takes 16 x 8 Y parts (2 x Y MMA tiles), accumulators started from C, the next
// part's C in flight meanwhile
template <int NT, int Y, class SM>
__device__ __forceinline__ void lu_update(const SM &S, int mt, int nt, double *C, long ldc) {
  constexpr int LDP = SM::LDP;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const int rb = (mt + 15) / 16, parts = rb * ((nt + 8 * Y - 1) / (8 * Y));
  const double *P = S.P + LPW;  // rows below the diagonal block
  auto load = [&](int s, double (&v)[2][Y][2]) {
    const int r0 = (s % rb) * 16 + g, c0 = (s / rb) * 8 * Y + 2 * t;
    const bool in0 = r0 < mt, in1 = r0 + 8 < mt;
    const double *Cp = C + r0 + (long)c0 * ldc;
#pragma unroll
    for (int y = 0; y < Y; y++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const bool in = s < parts && c0 + 8 * y + e < nt;
        const double *q = Cp + (8 * y + e) * ldc;
        v[0][y][e] = in && in0 ? q[0] : 0.0;
        v[1][y][e] = in && in1 ? q[8] : 0.0;
      }
  };
  double nx[2][Y][2];
  load(warp, nx);
#pragma unroll 1
  for (int s = warp; s < parts; s += NT / 32) {
    const int r0 = (s % rb) * 16 + g, c0 = (s / rb) * 8 * Y;
    const double *Pr = P + r0 + t * LDP, *Ur = S.U + (c0 + g) * LU_LDU + t;
    double acc[2][Y][2];
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
      for (int y = 0; y < Y; y++) {
        acc[x][y][0] = nx[x][y][0];
        acc[x][y][1] = nx[x][y][1];
      }
    load(s + NT / 32, nx);
#pragma unroll
    for (int q = 0; q < LPW; q += 4) {
      double av[2], bv[Y];
      av[0] = -Pr[q * LDP];          // rows past mt and columns past nt: not stored
      av[1] = -Pr[q * LDP + 8];
#pragma unroll
      for (int y = 0; y < Y; y++) bv[y] = Ur[8 * y * LU_LDU + q];
#pragma unroll
      for (int x = 0; x < 2; x++)
#pragma unroll
        for (int y = 0; y < Y; y++) cholb::dmma_8x8x4(acc[x][y], av[x], bv[y]);
    }
    const bool in0 = r0 < mt, in1 = r0 + 8 < mt;
    double *Cp = C + r0 + (long)(c0 + 2 * t) * ldc;
#pragma unroll
    for (int y = 0; y < Y; y++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const bool in = c0 + 8 * y + 2 * t + e < nt;
        double *q = Cp + (8 * y + e) * ldc;
        if (in && in0) q[0] = acc[0][y][e];
        if (in && in1) q[8] = acc[1][y][e];
      }
  }
}

}  // namespace atlb
