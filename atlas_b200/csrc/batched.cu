// Batched factorizations and solves of many small, uneven-size systems.  No
// counterpart in the reference (ATLAS factors one matrix per call); the
// per-problem arithmetic is that of ATL_potrfL / ATL_getf2 / ATL_potrs /
// ATL_getrs on a single small matrix.
//
// Persistent launches: CTAs pull problem indices from an atomic counter over
// a work list sorted by decreasing size (largest first, so the tail of a
// launch is made of small problems), and each problem is handled entirely by
// one CTA.  Cholesky: 16 x 16 tiles in shared memory, right-hand sides carried
// through the factorization, one launch per size bucket.  LU: 16-column
// pivoted panels in registers, the trailing update on the FP64 tensor cores in
// global memory, right-hand sides carried along too.  Nothing waits on another
// CTA, so a launch cannot stall.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstring>
#include <vector>
#include "common.cuh"
#include "chol_blocks.cuh"
#include "chol_tiles.cuh"
#include "kernels.h"
#include "lu_panel.cuh"
#include "staging.h"
#include "../../include/atlas_b200.h"

namespace atlb {
namespace {

constexpr int MAXN = 256;

struct Prob {
  double *A;
  double *B;
  int *ipiv;
  int n, lda, ldb, nrhs;
};

// ---------------------------------------------------------------- Cholesky

// Batched Cholesky + solve: each CTA takes whole problems off the list, the
// matrix as 16 x 16 tiles in shared memory (chol_tiles.cuh).  One launch per
// size bucket, because the shared memory a problem needs grows with its
// order: small orders then run many to an SM, which hides the chain of
// columns that bounds a single factorization.  The buckets (tiles per side,
// threads, CTAs per SM) end at the largest sizes at which one, two, four and
// eight CTAs fit the SM's 227 KB.
//
// 10,000 problems of orders 8..256 (mean 132) with 4 right-hand sides, B200:
// 17.5 ms before (panels in shared memory, the trailing matrix in L2, the
// right-hand sides solved one after another with loads of L on the chain),
// 2.9 ms now; the bytes of A and B would take 0.3 ms, the flops 0.5 ms.
template <int NT, int NBMAX>
struct PosvSmem {
  cholt::Shared<NBMAX> S;
  double rhs[NBMAX * cholt::RTILE];
  double pool[cholt::pool_tiles_upto(NBMAX, true) * cholt::TILE];
};

template <int NT, int NBMAX, int MINB>
__global__ void __launch_bounds__(NT, MINB)
batched_posv_kernel(const Prob *__restrict__ probs, const int *__restrict__ order, const int *__restrict__ range,
                    int *__restrict__ next, int *__restrict__ info) {
  extern __shared__ __align__(16) double sm[];
  auto &W = *reinterpret_cast<PosvSmem<NT, NBMAX> *>(sm);
  __shared__ int s_p;
  const int tid = threadIdx.x, end = range[1];
  while (true) {
    if (tid == 0) {
      const int t = range[0] + atomicAdd(next, 1);
      s_p = t < end ? order[t] : -1;
    }
    __syncthreads();
    const int p = s_p;
    if (p < 0) return;
    const Prob pr = probs[p];
    int fail = 0;
    if (pr.n > 0) {
      fail = cholt::factor<NT, false>(pr.n, pr.A, pr.lda, pr.B, pr.ldb, min(pr.nrhs, cholt::RHS), W.pool, W.rhs, W.S);
      if (!fail) cholt::solve<NT>(pr.n, pr.A, pr.lda, pr.B, pr.ldb, pr.nrhs, W.pool, W.rhs, W.S);
    }
    if (tid == 0) info[p] = fail;
    __syncthreads();
  }
}

// ---------------------------------------------------------------- LU

// Blocked LU with partial pivoting of one problem by one CTA, ATL_getrfC's
// right-looking step on panels of 16 columns, the trailing matrix in place in
// global memory (L2-resident at these orders):
//   1. the panel is factored in registers, one row per thread.  A column
//      costs one barrier: every warp's best row (largest |value|, lowest
//      current position on ties = cblas_idamax / ATL_getf2) goes to shared
//      memory before it, every thread picks the winner after it.  Rows do not
//      move: each carries its current position;
//   2. one thread per column right of the panel, right-hand sides included,
//      applies the panel's interchanges (only the top 16 rows and the pivot
//      rows change: one gather, one scatter) and solves U12 = L11^-1 A12 in
//      registers;
//   3. A22 -= L21 U12 on the FP64 tensor cores, L21 and U12 from shared
//      memory, the next part of A22 loaded under the products.
// The interchanges of the columns left of the panels wait until the end, where
// they are composed: applied panel by panel they moved as many bytes as step 2,
// a sector per entry (11.1 ms, with step 2's top rows read column by column).
// Up to eight right-hand sides ride along in shared memory, which makes the
// forward substitution part of the factorization.  What bounds it: the chain
// of columns (about 16 x 500 cycles a panel) and the L2 round trips of steps
// 2 and 3, so several CTAs share an SM: buckets of orders <= 64, 128, 256
// with 64, 128, 256 threads.
//
// 10,000 problems of orders 8..256 with one right-hand side, B200: getrf and
// getrs kernels 14.5 + 3.0 ms before (two barriers and a shared-memory rank-1
// update per column, interchanges and U12 as separate passes, a solve with
// loads of the factor on its chain), 9.6 ms now for both.
constexpr int LU_RHS = 8;       // right-hand sides carried along
constexpr int DLD = LPW + 1;

template <int NT>  // threads = largest order
struct LuSmem {
  static constexpr int LDP = NT + 4;  // 4 (mod 16): the MMA's 8 x 4 fragments fall in distinct banks
  double P[LPW * LDP];                // the factored panel, rows at their final places
  double U[NT * LU_LDU];
  double xs[LU_RHS * NT];             // right-hand sides
  double cand[2][NT / 32][LPW];       // per-warp candidate rows, by column parity
  unsigned long long ckey[2][NT / 32];
  int cpos[2][NT / 32];
  double D[2][LPW * DLD];             // diagonal blocks of the solves, D(r, q) at q * DLD + r
  int from[LPW], to[LPW];             // row whose content ends at q; where row q's content ends
  int piv[NT];                        // ipiv
  int fail;
};

// the factorization of one problem, S.xs (nr right-hand sides, row i of
// column r at r * NT + i) becoming L^-1 P b; returns the first zero pivot
// (1-based) or 0 and completes either way (LAPACK getrf semantics)
template <int NT>
__device__ __forceinline__ int lu_factor(const Prob &pr, int nr, LuSmem<NT> &S) {
  constexpr int LDP = LuSmem<NT>::LDP;
  const int tid = threadIdx.x, n = pr.n;
  double *A = pr.A;
  const long lda = pr.lda;
  if (tid == 0) S.fail = 0;
#pragma unroll 1
  for (int j = 0; j < n; j += LPW) {
    const int jb = min(LPW, n - j), m = n - j, nt = m - jb;
    double a[LPW];
#pragma unroll
    for (int k = 0; k < LPW; k++) a[k] = (tid < m && k < jb) ? A[j + tid + (long)(j + k) * lda] : 0.0;
    if (tid < LPW) {  // identity where the panel has fewer rows
      S.from[tid] = tid;
      S.to[tid] = tid;
    }
    __syncthreads();
    const int pos = lu_panel<NT, false>(S, a, m, jb, j);
#pragma unroll
    for (int k = 0; k < LPW; k++) a[k] = (tid < m && k < jb) ? S.P[k * LDP + tid] : 0.0;
    __syncthreads();
    if (tid < m) {
#pragma unroll
      for (int k = 0; k < LPW; k++) {
        S.P[k * LDP + pos] = a[k];
        if (k < jb) A[j + pos + (long)(j + k) * lda] = a[k];
      }
      if (pos < LPW) S.from[pos] = tid;
      if (tid < LPW) S.to[tid] = pos;
    }
    __syncthreads();
    // step 2: the columns right of the panel and the right-hand sides.  Their
    // top 16 rows come to U and go back from it 16 rows at a time; a column's
    // thread touches global memory only for the pivot rows below them.
    double *R = A + j + (long)(j + jb) * lda;
    for (int e = tid; e < nt * LPW; e += NT) {  // nt > 0: the panel has 16 columns
      const int q = e & (LPW - 1), k = e / LPW;
      S.U[k * LU_LDU + q] = R[q + k * lda];
    }
    __syncthreads();
#pragma unroll 1
    for (int cc = tid; cc < nt + nr; cc += NT) {
      const bool rhs = cc >= nt;
      double *col = rhs ? S.xs + (cc - nt) * NT + j : R + cc * lda, *u = rhs ? col : S.U + cc * LU_LDU;
      double x[LPW];  // shifted below: x[0] is the current row
#pragma unroll
      for (int q = 0; q < LPW; q++) {
        const int from = S.from[q];
        x[q] = q >= jb ? 0.0 : from < LPW ? u[from] : col[from];
      }
#pragma unroll 4
      for (int q = 0; q < LPW; q++) {
        const int to = S.to[q];
        if (to >= LPW) col[to] = u[q];
      }
#pragma unroll 1
      for (int q = 0; q < jb; q++) {
        const double v = x[0];
        u[q] = v;
        const double *l = S.P + q * LDP + q;
#pragma unroll
        for (int r = 1; r < LPW; r++) x[r - 1] = fma(-l[r], v, x[r]);
      }
    }
    __syncthreads();
    for (int e = tid; e < nt * LPW; e += NT) {
      const int q = e & (LPW - 1), k = e / LPW;
      R[q + k * lda] = S.U[k * LU_LDU + q];
    }
    __syncthreads();
    if (nt > 0) {
      if (tid >= LPW && tid < m)  // the right-hand sides' rows below the panel
#pragma unroll 1
        for (int r = 0; r < nr; r++) {
          double y = S.xs[r * NT + j + tid];
#pragma unroll
          for (int q = 0; q < LPW; q++) y = fma(-S.P[q * LDP + tid], S.xs[r * NT + j + q], y);
          S.xs[r * NT + j + tid] = y;
        }
      lu_update<NT, 4>(S, nt, nt, A + (j + jb) + (long)(j + jb) * lda, lda);
    }
    __syncthreads();
  }
  if (tid < n) pr.ipiv[tid] = S.piv[tid];
  // The interchanges of the columns left of each panel, all at once: `src` is
  // the row whose entry ends in this thread's row, composed from the last panel
  // back; every panel's multipliers are read and written once, in whole rows.
  int src = tid;
#pragma unroll 1
  for (int j = (n - 1) / LPW * LPW; j > 0; j -= LPW) {  // panel j moves the rows of panel j - 16
#pragma unroll 1
    for (int c = min(LPW, n - j) - 1; c >= 0; c--) {
      const int p = S.piv[j + c];
      src = src == j + c ? p : src == p ? j + c : src;
    }
    double *L = A + (long)(j - LPW) * lda;
    const bool in = tid >= j && tid < n;
    if (in)
#pragma unroll
      for (int q = 0; q < LPW; q++) S.P[q * LDP + tid] = L[tid + q * lda];
    __syncthreads();
    if (in && src != tid)
#pragma unroll
      for (int q = 0; q < LPW; q++) L[tid + q * lda] = S.P[q * LDP + src];
    __syncthreads();
  }
  return S.fail;
}

// v / d from r = 1 / d: v r corrected by its residual, which an FMA gives without
// rounding; correctly rounded where nothing over- or underflows on the way (P.
// Markstein, Computation of elementary functions on the IBM RISC System/6000
// processor, IBM J. Res. Dev. 34, 1990).  Operands far from one are divided.  On a
// substitution's chain a division is the longest link (10,000 problems of order 8
// with 32 right-hand sides: 650 us by v r alone, 989 divided, 694 so).
__device__ __forceinline__ bool mid_range(double x) { return fabs(x) > 1e-150 && fabs(x) < 1e150; }
__device__ __forceinline__ double quotient(double v, double d, double r) {
  const double q = v * r;
  return mid_range(v) ? fma(fma(-q, d, v), r, q) : v / d;
}

// U x = y (UPPER) or L x = y (unit lower) in place on nr <= 8 right-hand
// sides in S.xs, panel by panel: the panel's 16 columns are in registers, one
// row per thread, loaded one panel ahead; one warp per right-hand side solves
// the diagonal block, then every thread updates its row.
template <int NT, bool UPPER>
__device__ __forceinline__ void lu_solve(const Prob &pr, int nr, LuSmem<NT> &S) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = pr.n, np = (n + LPW - 1) / LPW;
  const double *A = pr.A;
  const long lda = pr.lda;
  auto load = [&](int s, double (&v)[LPW]) {
    const int j = (UPPER ? np - 1 - s : s) * LPW, jb = min(LPW, n - j);
    const bool in = s < np && tid < n && (UPPER ? tid < j + jb : tid >= j);
#pragma unroll
    for (int q = 0; q < LPW; q++) v[q] = in && q < jb ? A[tid + (long)(j + q) * lda] : 0.0;
    if (in && tid >= j && tid < j + jb) {
#pragma unroll
      for (int q = 0; q < LPW; q++) S.D[s & 1][q * DLD + tid - j] = v[q];
    }
  };
  double u[LPW];
  load(0, u);
#pragma unroll 1
  for (int s = 0; s < np; s++) {
    const int j = (UPPER ? np - 1 - s : s) * LPW, jb = min(LPW, n - j);
    __syncthreads();  // D and the rows updated by the last panel are in place
    double nx[LPW];
    load(s + 1, nx);
#pragma unroll 1
    for (int r = warp; r < nr; r += NT / 32) {
      const int c = lane & 15;
      double v = c < jb ? S.xs[r * NT + j + c] : 0.0;
      const double *d = S.D[s & 1] + c;  // D(c, q) at q * DLD + c
      const double piv = UPPER && c < jb ? d[c * DLD] : 1.0, ri = UPPER ? 1.0 / piv : 1.0;
      const bool mid = mid_range(piv);
      int q = UPPER ? jb - 1 : 0;
      double dn = d[q * DLD];
#pragma unroll 1
      for (int i = 0; i < jb; i++) {
        const double dq = dn;
        const int qn = UPPER ? max(q - 1, 0) : min(q + 1, LPW - 1);
        dn = d[qn * DLD];  // one step ahead of the chain
        if (UPPER && c == q) v = mid ? quotient(v, piv, ri) : v / piv;
        const double xq = __shfl_sync(0xffffffffu, v, q);
        if (UPPER ? c < q : c > q) v = fma(-dq, xq, v);
        q = qn;
      }
      if (lane < jb) S.xs[r * NT + j + c] = v;
    }
    __syncthreads();
    if (tid < n && (UPPER ? tid < j : tid >= j + jb))
#pragma unroll 1
      for (int r = 0; r < nr; r++) {
        double y = S.xs[r * NT + tid];
#pragma unroll
        for (int q = 0; q < LPW; q++)
          if (q < jb) y = fma(-u[q], S.xs[r * NT + j + q], y);
        S.xs[r * NT + tid] = y;
      }
#pragma unroll
    for (int q = 0; q < LPW; q++) u[q] = nx[q];
  }
  __syncthreads();
}

template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
batched_gesv_kernel(const Prob *__restrict__ probs, const int *__restrict__ order, const int *__restrict__ range,
                    int *__restrict__ next, int *__restrict__ info) {
  extern __shared__ __align__(16) double sm[];
  LuSmem<NT> &S = *reinterpret_cast<LuSmem<NT> *>(sm);
  __shared__ int s_p;
  const int tid = threadIdx.x, end = range[1];
  while (true) {
    if (tid == 0) {
      const int t = range[0] + atomicAdd(next, 1);
      s_p = t < end ? order[t] : -1;
    }
    __syncthreads();
    const int p = s_p;
    if (p < 0) return;
    const Prob pr = probs[p];
    int fail = 0;
    if (pr.n > 0) {
      const int n = pr.n, nr = min(pr.nrhs, LU_RHS);
#pragma unroll 1
      for (int r = 0; r < nr; r++)
        if (tid < n) S.xs[r * NT + tid] = pr.B[tid + (long)r * pr.ldb];
      fail = lu_factor<NT>(pr, nr, S);
      if (!fail)
#pragma unroll 1
        for (int r0 = 0; r0 < pr.nrhs; r0 += LU_RHS) {
          const int nc = min(LU_RHS, pr.nrhs - r0);
          double *B = pr.B + (long)r0 * pr.ldb;
          if (r0 > 0) {  // the columns that did not ride along
#pragma unroll 1
            for (int r = 0; r < nc; r++)
              if (tid < n) S.xs[r * NT + tid] = B[tid + (long)r * pr.ldb];
            __syncthreads();
            if (tid < nc)
#pragma unroll 1
              for (int k = 0; k < n; k++) {
                const int q = pr.ipiv[k];
                const double t0 = S.xs[tid * NT + k];
                S.xs[tid * NT + k] = S.xs[tid * NT + q];
                S.xs[tid * NT + q] = t0;
              }
            lu_solve<NT, false>(pr, nc, S);
          }
          lu_solve<NT, true>(pr, nc, S);
#pragma unroll 1
          for (int r = 0; r < nc; r++)
            if (tid < n) B[tid + (long)r * pr.ldb] = S.xs[r * NT + tid];
          __syncthreads();
        }
    }
    if (tid == 0) info[p] = fail;
    __syncthreads();
  }
}

// ---------------------------------------------------------------- host side

struct BatchBufs {
  Prob *probs;
  int *order, *next, *info;
  int *horder, *hnext;   // the pinned copies of order and next
  unsigned char *h, *d;  // pinned staging copy of the problem list, its device copy
  size_t bytes;          // bytes the upload copies
};

// The problem list, sorted by decreasing order, written into the pinned
// staging buffer (host side, every call); enqueue_upload() copies it to the
// device on the stream (a node of the captured graph on replays).
BatchBufs prepare(const std::vector<Prob> &P, int slot_p) {
  const int count = (int)P.size();
  std::vector<int> order(count);
  for (int i = 0; i < count; i++) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return P[a].n > P[b].n; });
  size_t bytes = sizeof(Prob) * count + sizeof(int) * (2 * count + 64);
  unsigned char *d = (unsigned char *)scratch(slot_p, bytes);
  unsigned char *h = (unsigned char *)pinned(slot_p, bytes);
  memcpy(h, P.data(), sizeof(Prob) * count);
  memcpy(h + sizeof(Prob) * count, order.data(), sizeof(int) * count);
  memset(h + sizeof(Prob) * count + sizeof(int) * count, 0, sizeof(int) * 64);
  BatchBufs b;
  b.probs = (Prob *)d;
  b.order = (int *)(d + sizeof(Prob) * count);
  b.next = b.order + count;
  b.info = b.next + 64;
  b.h = h;
  b.horder = (int *)(h + sizeof(Prob) * count);
  b.hnext = b.horder + count;
  b.d = d;
  b.bytes = bytes - sizeof(int) * count;
  return b;
}

void enqueue_upload(const BatchBufs &b, cudaStream_t st) {
  ATLB_CUDA_CHECK(cudaMemcpyAsync(b.d, b.h, b.bytes, cudaMemcpyHostToDevice, st));
}

template <int NT, int NBMAX, int MINB>
void launch_posv(const BatchBufs &b, int bucket, cudaStream_t st) {
  constexpr int smem = (int)sizeof(PosvSmem<NT, NBMAX>);
  static_assert(MINB * (smem + 1024 + 16) <= 228 * 1024, "the bucket's CTAs do not fit an SM");
  static bool configured = false;
  if (!configured) {
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(batched_posv_kernel<NT, NBMAX, MINB>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(batched_posv_kernel<NT, NBMAX, MINB>,
                                         cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    configured = true;
  }
  batched_posv_kernel<NT, NBMAX, MINB><<<num_sms() * MINB, NT, smem, st>>>(b.probs, b.order, b.next + 8 + 2 * bucket,
                                                                          b.next + bucket, b.info);
  ATLB_CUDA_CHECK(cudaGetLastError());
}

template <int NT, int MINB>
void launch_gesv(const BatchBufs &b, int bucket, cudaStream_t st) {
  constexpr int smem = (int)sizeof(LuSmem<NT>);
  static_assert(MINB * (smem + 1024 + 16) <= 228 * 1024, "the bucket's CTAs do not fit an SM");
  static bool configured = false;
  if (!configured) {
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(batched_gesv_kernel<NT, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem));
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(batched_gesv_kernel<NT, MINB>,
                                         cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    configured = true;
  }
  batched_gesv_kernel<NT, MINB><<<num_sms() * MINB, NT, smem, st>>>(b.probs, b.order, b.next + 8 + 2 * bucket,
                                                                   b.next + bucket, b.info);
  ATLB_CUDA_CHECK(cudaGetLastError());
}

// launch(bucket, stream) for each bucket in use, largest orders first: the first on
// st, the others one after another on a second stream beside it.  In a row, each
// bucket waited for the slowest problem of the one before, which for some hundred
// problems is most of the time (500 of orders 8..256, LU only: 967 us in a row, 658 so;
// 400 of orders 40..140: 571 and 360).
template <class Launch>
void launch_buckets(unsigned used, cudaStream_t st, Launch launch) {
  const bool several = (used & (used - 1)) != 0;
  cudaStream_t second = st;
  if (several) {
    second = copy_stream();
    ATLB_CUDA_CHECK(cudaEventRecord(side_event(6), st));
    ATLB_CUDA_CHECK(cudaStreamWaitEvent(second, side_event(6), 0));
  }
  bool first = true;
  for (int q = 0; used >> q; q++)
    if (used >> q & 1) {
      launch(q, first ? st : second);
      first = false;
    }
  if (several) {
    ATLB_CUDA_CHECK(cudaEventRecord(side_event(7), second));
    ATLB_CUDA_CHECK(cudaStreamWaitEvent(st, side_event(7), 0));
  }
}

// Cuts the sorted list into buckets of orders above lower[0], lower[1], ..;
// returns the mask of those in use.
unsigned bucket_ranges(const std::vector<Prob> &P, const BatchBufs &b, const int *lower, int nbuckets) {
  int *range = b.hnext + 8, at = 0;
  unsigned used = 0;
  for (int q = 0; q < nbuckets; q++) {
    range[2 * q] = at;
    while (at < (int)P.size() && P[b.horder[at]].n > lower[q]) at++;
    range[2 * q + 1] = at;
    if (at > range[2 * q]) used |= 1u << q;
  }
  return used;
}

}  // namespace

// One batched Cholesky + solve: upload, one launch per size bucket in use, info back to
// info_out (pinned).  The launch sequence depends only on the batch's shape
// and the buffers, so it is replayed from a CUDA graph from the third call on
// (run_graph): the problem list itself travels in the captured copy.
void batched_posv_dev(const std::vector<Prob> &P, int *info_out, cudaStream_t st) {
  const int count = (int)P.size();
  if (!count) return;
  BatchBufs b = prepare(P, kSlotBatch0);
  static const int lower[4] = {11 * cholt::TB, 7 * cholt::TB, 3 * cholt::TB, -1};
  const unsigned used = bucket_ranges(P, b, lower, 4);
  const std::vector<unsigned long long> key = {0xBA7C0001ull, (unsigned long long)tune_generation(),
      (unsigned long long)count, (unsigned long long)used, (unsigned long long)(uintptr_t)b.d,
      (unsigned long long)(uintptr_t)b.h, (unsigned long long)(uintptr_t)info_out,
      (unsigned long long)(uintptr_t)st};
  run_graph(key, st, [&]() {
    enqueue_upload(b, st);
    launch_buckets(used, st, [&](int q, cudaStream_t s) {
      if (q == 0) launch_posv<256, 16, 1>(b, 0, s);
      else if (q == 1) launch_posv<256, 11, 2>(b, 1, s);
      else if (q == 2) launch_posv<128, 7, 4>(b, 2, s);
      else launch_posv<64, 3, 8>(b, 3, s);
    });
    ATLB_CUDA_CHECK(cudaMemcpyAsync(info_out, b.info, sizeof(int) * count, cudaMemcpyDeviceToHost, st));
  });
}

// Batched LU (+ the solve of each problem's right-hand sides), the same way.
void batched_gesv_dev(const std::vector<Prob> &P, int *info_out, cudaStream_t st) {
  const int count = (int)P.size();
  if (!count) return;
  BatchBufs b = prepare(P, kSlotBatch0);
  static const int lower[3] = {128, 64, -1};
  const unsigned used = bucket_ranges(P, b, lower, 3);
  const std::vector<unsigned long long> key = {0xBA7C0002ull,
      (unsigned long long)tune_generation(), (unsigned long long)count, (unsigned long long)used,
      (unsigned long long)(uintptr_t)b.d, (unsigned long long)(uintptr_t)b.h,
      (unsigned long long)(uintptr_t)info_out, (unsigned long long)(uintptr_t)st};
  run_graph(key, st, [&]() {
    enqueue_upload(b, st);
    launch_buckets(used, st, [&](int q, cudaStream_t s) {
      if (q == 0) launch_gesv<256, 2>(b, 0, s);
      else if (q == 1) launch_gesv<128, 4>(b, 1, s);
      else launch_gesv<64, 7>(b, 2, s);
    });
    ATLB_CUDA_CHECK(cudaMemcpyAsync(info_out, b.info, sizeof(int) * count, cudaMemcpyDeviceToHost, st));
  });
}

}  // namespace atlb

using namespace atlb;

extern "C" {

// Batched Cholesky factor + solve of `count` independent SPD systems (lower
// triangle referenced, column-major): A[i] (n[i] x n[i], lda[i]) and B[i]
// (n[i] x nrhs[i], ldb[i]) are DEVICE pointers; on return A[i] holds L and
// B[i] the solution, info[i] (host array) the potrf info.  Orders up to 256.  Returns 0 or a negative argument position.
int atlb_dposv_batched(int count, const int *n, double *const *A, const int *lda, double *const *B,
                       const int *ldb, const int *nrhs, int *info) {
  if (count < 0) return -1;
  if (count == 0) return 0;
  std::vector<Prob> P(count);
  for (int i = 0; i < count; i++) {
    if (n[i] < 0 || n[i] > MAXN) return -2;
    if (lda[i] < std::max(1, n[i])) return -4;
    if (ldb[i] < std::max(1, n[i])) return -6;
    if (nrhs[i] < 0) return -7;
    P[i] = {A[i], B[i], nullptr, n[i], lda[i], ldb[i], nrhs[i]};
  }
  cudaStream_t st = stream();
  int *hinfo = (int *)pinned(kSlotBatch1, sizeof(int) * count);
  batched_posv_dev(P, hinfo, st);
  sync_stream(st);
  memcpy(info, hinfo, sizeof(int) * count);
  return 0;
}

// Batched LU with partial pivoting (+ optional solve when B is non-NULL):
// device pointers as above; ipiv[i] device int arrays of n[i] entries
// (0-based), info[i] host.  Orders up to 256.
int atlb_dgesv_batched(int count, const int *n, double *const *A, const int *lda, int *const *ipiv,
                       double *const *B, const int *ldb, const int *nrhs, int *info) {
  if (count < 0) return -1;
  if (count == 0) return 0;
  std::vector<Prob> P(count);
  for (int i = 0; i < count; i++) {
    if (n[i] < 0 || n[i] > MAXN) return -2;
    if (lda[i] < std::max(1, n[i])) return -4;
    if (B && (ldb[i] < std::max(1, n[i]) || nrhs[i] < 0)) return -7;
    P[i] = {A[i], B ? B[i] : nullptr, ipiv[i], n[i], lda[i], B ? ldb[i] : 1, B ? nrhs[i] : 0};
  }
  cudaStream_t st = stream();
  int *hinfo = (int *)pinned(kSlotBatch1, sizeof(int) * count);
  batched_gesv_dev(P, hinfo, st);
  sync_stream(st);
  memcpy(info, hinfo, sizeof(int) * count);
  return 0;
}

// Batched LU with partial pivoting only (LAPACK getrf semantics per problem:
// A[i] overwritten by L\U, ipiv[i] 0-based device arrays, info[i] host).
int atlb_dgetrf_batched(int count, const int *n, double *const *A, const int *lda, int *const *ipiv, int *info) {
  return atlb_dgesv_batched(count, n, A, lda, ipiv, nullptr, nullptr, nullptr, info);
}

}  // extern "C"
