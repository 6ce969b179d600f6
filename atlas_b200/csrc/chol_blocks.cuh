// Blocked Cholesky in shared memory, for one CTA of 256 threads: the FP32
// potrf (chol.cu) factors its diagonal blocks with it (FP64: chol_tiles.cuh).
// Also the FP64 MMA of the other kernels.
#pragma once
#include <cuda_runtime.h>

namespace atlb {
namespace cholb {

// C (rows < mt, columns < nc <= mt, lower part i >= k) -= P P^T, P = mt x jb
// (ld lds, shared memory); C in shared or global memory (ldc).  16 x 16
// threads, 4 x 4 register tiles over 64 x 64 blocks of the lower trapezoid.
template <typename T, typename CT>
__device__ __forceinline__ void syrk_lower_update(int mt, int nc, int jb, const T *P, int lds, CT *C, long ldc) {
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  for (int ib = 0; ib < mt; ib += 64)
    for (int kb = 0; kb <= ib && kb < nc; kb += 64) {
      T acc[4][4];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) acc[a][b] = T(0);
      for (int q = 0; q < jb; q++) {
        T pi[4], pk[4];
#pragma unroll
        for (int a = 0; a < 4; a++) {
          const int i = ib + tx + 16 * a;
          pi[a] = i < mt ? P[i + q * lds] : T(0);
        }
#pragma unroll
        for (int b = 0; b < 4; b++) {
          const int k = kb + ty + 16 * b;
          pk[b] = k < nc ? P[k + q * lds] : T(0);
        }
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
          for (int b = 0; b < 4; b++) acc[a][b] = fma(pi[a], pk[b], acc[a][b]);
      }
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) {
          const int i = ib + tx + 16 * a, k = kb + ty + 16 * b;
          if (i < mt && k < nc && k <= i) C[i + (long)k * ldc] -= acc[a][b];
        }
    }
}

// Leading dimension for an order-n matrix in shared memory: the smallest value
// >= n that is 8 (mod 16).
__host__ __device__ constexpr int ld_for(int n) { return (n + 7) / 16 * 16 + 8; }

// d += a b on one m8n8k4 FP64 tensor-core tile (PTX mma.m8n8k4 .f64
// fragments: a = A[g][t], b = B[t][g], d = D[g][2t..2t+1], g = lane / 4,
// t = lane % 4)
__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Cholesky of the jb <= 16 columns of the m x jb panel at s (ld lds, rows
// from the panel's diagonal).  Warp 0 factors the jb x jb diagonal block:
// lane i holds row i in registers and every lane keeps its own copy of the
// jb diagonal entries, so the column-to-column chain (diagonal -> 1/sqrt ->
// multipliers -> next diagonal) has no shuffle and no block barrier; each
// finished column goes to shared memory, where the lanes read the
// multipliers back after a warp barrier.  Then every thread solves rows of
// L21 = A21 L11^-T on its own.  Right-looking order within each row, as the
// unblocked algorithm: column c is scaled by 1/sqrt(d_c), then its multiple
// is subtracted from columns c+1.. .  JB > 0 fixes jb at compile time.
// Returns 0 or the first non-positive pivot (1-based, panel-relative), the
// same in every thread; the columns before it are then factored and stored,
// the rest of the panel is not.
template <typename T, int JB>
__device__ int chol_panel_w(T *s, int lds, int m, int jb_) {
  __shared__ T s_rinv[16];
  __shared__ int s_fail;
  const int jb = JB ? JB : jb_;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (tid < 32) {
    const int i = tid;
    T r[16], dd[16];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      r[k] = (i < jb && k < jb && k <= i) ? s[i + k * lds] : T(0);
      dd[k] = k < jb ? s[k + k * lds] : T(1);
    }
    int fail = 0;
#pragma unroll
    for (int c = 0; c < 16; c++) {
      if (c >= jb) continue;
      const T d = dd[c];
      if (!(d > T(0)) && !fail) fail = c + 1;  // later columns run on, unstored
      const T ri = rsqrt(d);
      const T l = (i == c ? d : r[c]) * ri;  // L[i][c] (zero above the diagonal)
      if (!fail && i >= c && i < jb) s[i + c * lds] = l;
      if (i == 0) s_rinv[c] = ri;
      __syncwarp();
#pragma unroll
      for (int k = c + 1; k < 16; k++) {
        if (k >= jb) continue;
        const T lk = fail ? T(0) : s[k + c * lds];
        dd[k] = fma(-lk, lk, dd[k]);
        if (i >= k) r[k] = fma(-l, lk, r[k]);
      }
    }
    if (i == 0) s_fail = fail;
  }
  __syncthreads();
  const int fail = s_fail;
  if (fail) {
    __syncthreads();  // s_fail read by all before a later call rewrites it
    return fail;
  }
  for (int i = jb + tid; i < m; i += nt) {
    T x[16];
#pragma unroll
    for (int c = 0; c < 16; c++) x[c] = c < jb ? s[i + c * lds] : T(0);
#pragma unroll
    for (int c = 0; c < 16; c++) {
      if (c >= jb) continue;
      x[c] = x[c] * s_rinv[c];
#pragma unroll
      for (int k = c + 1; k < 16; k++)
        if (k < jb) x[k] = fma(-x[c], s[k + c * lds], x[k]);
    }
#pragma unroll
    for (int c = 0; c < 16; c++)
      if (c < jb) s[i + c * lds] = x[c];
  }
  __syncthreads();
  return 0;
}

template <typename T>
__device__ int chol_panel16(T *s, int lds, int m, int jb) {
  return jb == 16 ? chol_panel_w<T, 16>(s, lds, m, jb) : chol_panel_w<T, 0>(s, lds, m, jb);
}

// Cholesky of the jb columns of the m x jb panel at s (ld lds, rows from the
// panel's diagonal): 16-column sub-panels, each followed by the update of the
// panel's columns right of it (a lower trapezoid).  Returns 0 or the first
// non-positive pivot (1-based, panel-relative), the same in every thread; on
// failure the panel is left partly factored.
template <typename T>
__device__ int chol_panel(T *s, int lds, int m, int jb) {
  for (int j = 0; j < jb; j += 16) {
    const int w = min(16, jb - j), rest = jb - j - w;
    T *P = s + j + j * lds;
    const int f = chol_panel16(P, lds, m - j, w);
    if (f) return j + f;
    if (rest > 0) {
      syrk_lower_update(m - j - w, rest, w, P + w, lds, P + w + w * lds, lds);
      __syncthreads();
    }
  }
  return 0;
}

// blocked right-looking Cholesky of an n x n lower matrix in shared memory
// (ld lds); returns 0 or the first non-positive pivot (1-based), the matrix
// then partly factored
template <typename T>
__device__ int chol_smem(T *s, int lds, int n) {
  return chol_panel(s, lds, n, n);
}

}  // namespace cholb
}  // namespace atlb
