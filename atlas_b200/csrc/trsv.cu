// Triangular solve for a few right-hand sides (FP32 <= 8, FP64 <= 16) in ONE launch.
//
// The recursive TRSM (trsm.cu) issues ~2n/64 launches, which for one
// right-hand side is all latency.  Here one CTA owns one 128-row block of
// the solution (two 64-row sub-blocks): it takes a ticket from an atomic
// counter (tickets are handed out in launch order, so every block it depends
// on is owned by a CTA that is already running and never waits on it) and
// accumulates the products with the solved blocks.  The blocks solved long
// ago are streamed in bulk: one warp looks up to 32 "done" flags at once
// and the CTA then runs through every block found done without waiting
// again; only the block just before it is awaited, with its matrix values
// already in registers.  The block is then solved by one product with the
// inverse of its 128 x 128 diagonal block (computed once per factor by
// trsv_inverse_dev, loaded into shared memory before any wait) and
// published.  In FP32 the block just before is not awaited through its flag:
// its x also goes out as (value, epoch) 64-bit words, each written by one
// single-copy-atomic store, and the next block polls those words directly --
// one round trip to L2 on the chain instead of fence, flag and data load (in
// FP64, with two words a value, that changed nothing).
// Every wait is bounded: after ~1 s the kernel reports it (wait_word()), stops
// waiting, and marks its block of x, and so all that follow from it, with NaN.  The
// launcher clears the ticket counter, the flags and the tagged words before
// each launch.
#include <algorithm>
#include "common.cuh"
#include "kernels.h"
#include "chol_blocks.cuh"

namespace atlb {
namespace {

constexpr int BS = 64;       // rows of a diagonal block (W's blocks)
constexpr int CB = 2 * BS;   // rows of one CTA's block
constexpr int TT = 512;      // threads: four per row of the CTA's block
constexpr int NQ = TT / CB;  // parts a row's dot products are split into
constexpr int PART = CB / NQ;  // columns of a solved block per thread

__device__ __forceinline__ uint64_t gtimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <typename T, int NR>
__global__ void __launch_bounds__(TT, 1)
trsv_kernel(int n, int nrhs, const T *__restrict__ Tp, long tr, long tc, int lower,
            const T *__restrict__ W, T *X, long ldx, int *counter, int *flags, int epoch, int *word,
            unsigned long long *xt) {
  extern __shared__ __align__(16) unsigned char trsv_smem[];
  T(*sW)[CB + 1] = reinterpret_cast<T(*)[CB + 1]>(trsv_smem);   // [CB]: the inverted diagonal block
  T(*sxd)[CB][NR] = reinterpret_cast<T(*)[CB][NR]>(sW + CB);    // x of a solved block, double-buffered
  T(*sb)[NR] = reinterpret_cast<T(*)[NR]>(sxd + 2);             // this block's b
  T(*sacc)[CB][NR] = reinterpret_cast<T(*)[CB][NR]>(sb + CB);   // [NQ]: the parts' sums
  __shared__ int s_bi, s_ready, s_late[2];
  const int tid = threadIdx.x, lane = tid & 31, nb = (n + CB - 1) / CB;
  if (tid == 0) {
    const int t = atomicAdd(counter, 1);
    s_bi = lower ? t : nb - 1 - t;
    s_late[0] = s_late[1] = 0;
  }
  __syncthreads();
  const int bi = s_bi, r0 = bi * CB, rows = min(CB, n - r0);
  // everything that does not depend on other blocks is fetched first
  {
    const T *Wb = W + (long)bi * CB * CB;  // column-major 128 x 128
    for (int base = tid; base < CB * CB; base += 8 * TT) {  // eight loads in flight per thread
      T v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = Wb[base + q * TT];
#pragma unroll
      for (int q = 0; q < 8; q++) sW[(base + q * TT) % CB][(base + q * TT) / CB] = v[q];
    }
  }
  for (int idx = tid; idx < CB * NR; idx += TT) {
    const int rr = idx % CB, q = idx / CB;
    sb[rr][q] = (rr < rows && q < nrhs) ? X[r0 + rr + (long)q * ldx] : T(0);
  }
  // thread (row, part): row of this block, columns part*PART .. +PART-1 of every solved block
  const int row = tid % CB, part = tid / CB;
  const T *trow = Tp + (long)(r0 + row) * tr;
  const int ndep = lower ? bi : nb - 1 - bi;
  T acc[NR], acc2[NR];  // even and odd columns: two independent FMA chains
#pragma unroll
  for (int q = 0; q < NR; q++) acc[q] = acc2[q] = T(0);
  auto give_up = [&]() {  // one thread: b, and with it x, becomes NaN
    report_lost_wait(word);
    for (int idx = 0; idx < CB * NR; idx++) sb[idx / NR][idx % NR] = (T)__longlong_as_double(-1LL);
  };
  auto wait_flag = [&](int bj) {
    const uint64_t t0 = gtimer();
    while (ld_acquire(flags + bj) != epoch) {
      if (gtimer() - t0 > 1000000000ull) { give_up(); break; }
    }
  };
  // x of block bj into sxd[buf] (all threads), then the products
  auto load_x = [&](int bj, int buf) {
    const int c0 = bj * CB;
    for (int idx = tid; idx < CB * NR; idx += TT) {
      const int cc = idx % CB, q = idx / CB;
      sxd[buf][cc][q] = (c0 + cc < n && q < nrhs) ? __ldcg(X + c0 + cc + (long)q * ldx) : T(0);
    }
  };
  // 1. solved blocks in bulk: all but the last dependency
  int d = 0, buf = 0;
  while (d < ndep - 1) {
    if (tid < 32) {
      // how many of the next blocks (up to 32, never the last one) are done
      const int dd = d + lane;
      const bool ok = dd < ndep - 1 && ld_acquire(flags + (lower ? dd : nb - 1 - dd)) == epoch;
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      const int ready = __ffs(~m) - 1;  // leading run of done blocks
      if (lane == 0) {
        if (ready == 0) wait_flag(lower ? d : nb - 1 - d);
        s_ready = ready == 0 ? 1 : ready;
      }
    }
    __syncthreads();
    const int nr = s_ready;
    for (int e = 0; e < nr; e++, d++) {
      const int bj = lower ? d : nb - 1 - d;
      const int c0 = bj * CB + part * PART, cols = min(PART, n - c0);
      // all of this thread's matrix loads in flight at once, issued before
      // the barrier: a CTA far down the triangle streams many blocks, and
      // this stream (not the chain of solves) bounds it when fewer loads
      // are in flight
      T tv[PART];
#pragma unroll
      for (int k = 0; k < PART; k++) tv[k] = (row < rows && k < cols) ? trow[(long)(c0 + k) * tc] : T(0);
      load_x(bj, buf);
      __syncthreads();
      const T(*xs)[NR] = sxd[buf] + part * PART;
#pragma unroll
      for (int k = 0; k < PART; k += 2)
#pragma unroll
        for (int q = 0; q < NR; q++) {
          acc[q] = fma(tv[k], xs[k][q], acc[q]);
          acc2[q] = fma(tv[k + 1], xs[k + 1][q], acc2[q]);
        }
      buf ^= 1;
    }
    __syncthreads();  // s_ready is read by every thread before it is rewritten
  }
  // 2. the block just before this one: its matrix values first, then the wait
  if (ndep > 0) {
    const int bj = lower ? ndep - 1 : nb - ndep;
    const int c0 = bj * CB + part * PART, cols = min(PART, n - c0);
    T tv[PART];
#pragma unroll
    for (int k = 0; k < PART; k++) tv[k] = (row < rows && k < cols) ? trow[(long)(c0 + k) * tc] : T(0);
    if constexpr (sizeof(T) == 4) {
      // FP32: x arrives as (value, epoch) 64-bit words, each written by one
      // single-copy-atomic store, so a word whose tag is current carries its
      // value: one round trip to L2 instead of flag, fence and data
      const uint64_t t0 = gtimer();
      int poll = 0;
      while (true) {
        bool ok = true;
        for (int idx = tid; idx < CB * NR; idx += TT) {
          const int cc = idx % CB, q = idx / CB;
          T v = T(0);
          if (bj * CB + cc < n && q < nrhs) {
            const unsigned long long w = __ldcg(xt + (long)(bj * CB + cc) * NR + q);
            ok = ok && (int)(w >> 32) == epoch;
            v = __uint_as_float((unsigned)(w & 0xffffffffu));
          }
          sxd[buf][cc][q] = v;
        }
        if (__syncthreads_and(ok)) break;
        if (s_late[poll & 1]) {  // thread 0's clock as of the poll before, so that all leave together
          if (tid == 0) give_up();
          break;
        }
        poll++;
        if (tid == 0 && gtimer() - t0 > 1000000000ull) s_late[poll & 1] = 1;
      }
    } else {
      if (tid == 0) wait_flag(bj);
      __syncthreads();
      load_x(bj, buf);
      __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < PART; k += 2)
#pragma unroll
      for (int q = 0; q < NR; q++) {
        acc[q] = fma(tv[k], sxd[buf][part * PART + k][q], acc[q]);
        acc2[q] = fma(tv[k + 1], sxd[buf][part * PART + k + 1][q], acc2[q]);
      }
  }
#pragma unroll
  for (int q = 0; q < NR; q++) sacc[part][row][q] = acc[q] + acc2[q];
  __syncthreads();
  for (int idx = tid; idx < CB * NR; idx += TT) {
    const int rr = idx % CB, q = idx / CB;
    T t = T(0);
#pragma unroll
    for (int p = 0; p < NQ; p++) t += sacc[p][rr][q];
    sb[rr][q] -= t;
  }
  __syncthreads();
  // 3. x = inv(T_bb) b: thread (row, part) sums over a quarter of the columns
  {
    T v[NR], v2[NR];
#pragma unroll
    for (int q = 0; q < NR; q++) v[q] = v2[q] = T(0);
#pragma unroll
    for (int c = part * PART; c < part * PART + PART; c += 2) {
      const T w = sW[row][c], w2 = sW[row][c + 1];
#pragma unroll
      for (int q = 0; q < NR; q++) {
        v[q] = fma(w, sb[c][q], v[q]);
        v2[q] = fma(w2, sb[c + 1][q], v2[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < NR; q++) sacc[part][row][q] = v[q] + v2[q];
  }
  __syncthreads();
  for (int idx = tid; idx < CB * NR; idx += TT) {
    const int rr = idx % CB, q = idx / CB;
    T t = T(0);
#pragma unroll
    for (int p = 0; p < NQ; p++) t += sacc[p][rr][q];
    if (rr < rows && q < nrhs) {
      X[r0 + rr + (long)q * ldx] = t;
      if constexpr (sizeof(T) == 4)
        xt[(long)(r0 + rr) * NR + q] =
            ((unsigned long long)(unsigned)epoch << 32) | (unsigned long long)__float_as_uint((float)t);
    }
  }
  __syncthreads();
  if (tid == 0) {  // the barrier orders every thread's x stores before this release
    __threadfence();
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(flags + bi), "r"(epoch) : "memory");
  }
}

// The same solve in FP64 for up to 8 NH right-hand sides, with the products on
// the FP64 tensor cores.  A chain step (the product with the block
// just before, then the one with the inverted diagonal block) is 128 x 128 x 8
// twice: with FMAs every term needs its x from shared memory (8192^2, 8
// right-hand sides: 13.5 us a block), while the MMA's n = 8 columns are the
// right-hand sides themselves and one fragment of x serves 8 rows.  Warp w
// owns rows 8 w .. 8 w + 7; its fragments of T come from global memory before
// the wait.  Two groups of columns share every fragment of T and the chain's
// latency, hence up to 16 per launch: 8192^2, 16 right-hand sides, one
// direction 472 us; with FMAs, eight at a time, 2 x 860.  The step is bound by
// its latency, so 1..4 right-hand sides, with most of the eight columns zero,
// take it too: both directions of 8192^2 in 764 us (FMAs: 2..4 1266), of 3000^2 in
// 298 (436), of 1000^2 in 144 (183).  One right-hand side keeps the FMAs where a
// column of T is contiguous in memory: their lanes run down it, while the fragments
// take eight rows of four columns (getrs, both factors, without transposition, 8192^2:
// 1106 us here, 862 with FMAs, 2000^2 304 and 249, 400^2 122 and 111; transposed 1096
// here and 1970 with FMAs, 307 and 503, 123 and 178), and over one or two blocks, where
// nothing chains (200^2: 80.7 us, here 84.4).
template <int NH>
__global__ void __launch_bounds__(TT, 1)
trsv_mma_kernel(int n, int nrhs, const double *__restrict__ Tp, long tr, long tc, int lower,
                const double *__restrict__ W, double *X, long ldx, int *counter, int *flags, int epoch, int *word) {
  constexpr int NR = 8 * NH, LX = NH == 1 ? 12 : 20, LW = CB + 4;  // fragments in distinct banks
  extern __shared__ __align__(16) unsigned char trsv_smem[];
  double *sW = reinterpret_cast<double *>(trsv_smem);  // W(r, c) at r * LW + c
  double *sx = sW + CB * LW;                           // x of a solved block (row k at k * LX), double-buffered
  double *sb = sx + 2 * CB * LX;                       // this block's b
  __shared__ int s_bi, s_ready;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = (n + CB - 1) / CB;
  const int g = lane >> 2, t = lane & 3;
  if (tid == 0) {
    const int k = atomicAdd(counter, 1);
    s_bi = lower ? k : nb - 1 - k;
  }
  __syncthreads();
  const int bi = s_bi, r0 = bi * CB, rows = min(CB, n - r0);
  {
    const double *Wb = W + (long)bi * CB * CB;
    for (int base = tid; base < CB * CB; base += 8 * TT) {
      double v[8];
#pragma unroll
      for (int q = 0; q < 8; q++) v[q] = Wb[base + q * TT];
#pragma unroll
      for (int q = 0; q < 8; q++) sW[(base + q * TT) % CB * LW + (base + q * TT) / CB] = v[q];
    }
  }
  for (int idx = tid; idx < CB * NR; idx += TT) {
    const int rr = idx % CB, q = idx / CB;
    sb[rr * LX + q] = (rr < rows && q < nrhs) ? X[r0 + rr + (long)q * ldx] : 0.0;
  }
  const int row = 8 * warp + g;
  const double *trow = Tp + (long)(r0 + row) * tr;
  const int ndep = lower ? bi : nb - 1 - bi;
  double acc[NH][2];
#pragma unroll
  for (int h = 0; h < NH; h++) acc[h][0] = acc[h][1] = 0.0;
  auto give_up = [&]() {  // one thread: b, and with it x, becomes NaN
    report_lost_wait(word);
    for (int idx = 0; idx < CB * LX; idx++) sb[idx] = __longlong_as_double(-1LL);
  };
  auto wait_flag = [&](int bj) {
    const uint64_t t0 = gtimer();
    while (ld_acquire(flags + bj) != epoch) {
      if (gtimer() - t0 > 1000000000ull) { give_up(); break; }
    }
  };
  auto load_t = [&](int bj, double (&a)[CB / 4]) {
    const int c0 = bj * CB;
#pragma unroll
    for (int k = 0; k < CB / 4; k++)
      a[k] = (row < rows && c0 + 4 * k + t < n) ? trow[(long)(c0 + 4 * k + t) * tc] : 0.0;
  };
  auto load_x = [&](int bj, int buf) {
    const int c0 = bj * CB;
    for (int idx = tid; idx < CB * NR; idx += TT) {
      const int cc = idx % CB, q = idx / CB;
      sx[buf * CB * LX + cc * LX + q] = (c0 + cc < n && q < nrhs) ? __ldcg(X + c0 + cc + (long)q * ldx) : 0.0;
    }
  };
  auto multiply = [&](const double (&a)[CB / 4], int buf) {
    const double *xs = sx + buf * CB * LX + t * LX + g;
#pragma unroll
    for (int k = 0; k < CB / 4; k++)
#pragma unroll
      for (int h = 0; h < NH; h++) cholb::dmma_8x8x4(acc[h], a[k], xs[4 * k * LX + 8 * h]);
  };
  // 1. solved blocks in bulk: all but the last dependency
  int d = 0, buf = 0;
  while (d < ndep - 1) {
    if (tid < 32) {
      const int dd = d + lane;
      const bool ok = dd < ndep - 1 && ld_acquire(flags + (lower ? dd : nb - 1 - dd)) == epoch;
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      const int ready = __ffs(~m) - 1;  // leading run of done blocks
      if (lane == 0) {
        if (ready == 0) wait_flag(lower ? d : nb - 1 - d);
        s_ready = ready == 0 ? 1 : ready;
      }
    }
    __syncthreads();
    const int nr = s_ready;
    for (int e = 0; e < nr; e++, d++) {
      const int bj = lower ? d : nb - 1 - d;
      double a[CB / 4];
      load_t(bj, a);
      load_x(bj, buf);
      __syncthreads();
      multiply(a, buf);
      buf ^= 1;
    }
    __syncthreads();  // s_ready is read by every thread before it is rewritten
  }
  // 2. the block just before this one: its matrix values first, then the wait
  if (ndep > 0) {
    const int bj = lower ? ndep - 1 : nb - ndep;
    double a[CB / 4];
    load_t(bj, a);
    if (tid == 0) wait_flag(bj);
    __syncthreads();
    load_x(bj, buf);
    __syncthreads();
    multiply(a, buf);
  } else {
    __syncthreads();  // sb is in place
  }
#pragma unroll
  for (int h = 0; h < NH; h++)
#pragma unroll
    for (int e = 0; e < 2; e++) sb[row * LX + 8 * h + 2 * t + e] -= acc[h][e];
  __syncthreads();
  // 3. x = inv(T_bb) b, the triangle's zero half left out
#pragma unroll
  for (int h = 0; h < NH; h++) acc[h][0] = acc[h][1] = 0.0;
  const int k0 = lower ? 0 : 2 * warp, k1 = lower ? 2 * warp + 2 : CB / 4;
#pragma unroll 4
  for (int k = k0; k < k1; k++) {
    const double w = sW[row * LW + 4 * k + t];
#pragma unroll
    for (int h = 0; h < NH; h++) cholb::dmma_8x8x4(acc[h], w, sb[(4 * k + t) * LX + 8 * h + g]);
  }
#pragma unroll
  for (int h = 0; h < NH; h++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int q = 8 * h + 2 * t + e;
      if (row < rows && q < nrhs) X[r0 + row + (long)q * ldx] = acc[h][e];
    }
  __syncthreads();
  if (tid == 0) {  // the barrier orders every thread's x stores before this release
    __threadfence();
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(flags + bi), "r"(epoch) : "memory");
  }
}

// The 128 x 128 diagonal blocks' inverses from the 64 x 64 ones (W64, as
// trinv_kernel leaves them): lower [W0 0; -W1 T10 W0  W1], upper
// [W0  -W0 T01 W1; 0 W1], with W1 = I when the last block has one sub-block.
// One CTA per block, the 128 x 128 block in shared memory: the off-diagonal
// quadrant first holds T's, then Y = T10 W0 (or T01 W1), then -W1 Y (or
// -W0 Y).  Written column-major, 128 x 128 per block.
template <typename T>
__global__ void __launch_bounds__(256)
trinv128_kernel(int n, const T *__restrict__ Tp, long tr, long tc, int lower, const T *__restrict__ W64,
                T *__restrict__ W128) {
  extern __shared__ __align__(16) unsigned char t128_smem[];
  T(*s)[CB + 1] = reinterpret_cast<T(*)[CB + 1]>(t128_smem);
  const int b = blockIdx.x, r0 = b * CB, tid = threadIdx.x;
  const int nsub = min(2, (n - r0 + BS - 1) / BS);
  for (int base = tid; base < CB * CB; base += 8 * 256) {  // eight loads in flight per thread
    T v[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int idx = base + 256 * q;
      const int i = idx % CB, k = idx / CB, qi = i / BS, qk = k / BS, ii = i % BS, kk = k % BS;
      v[q] = T(0);
      if (qi == qk) {
        if (qi < nsub) v[q] = W64[(long)(2 * b + qi) * BS * BS + ii + kk * BS];
        else v[q] = ii == kk ? T(1) : T(0);
      } else if (lower ? qi == 1 : qi == 0) {  // the triangle's off-diagonal quadrant
        const int gi = r0 + i, gk = r0 + k;
        if (gi < n && gk < n) v[q] = Tp[gi * tr + gk * tc];
      }
    }
#pragma unroll
    for (int q = 0; q < 8; q++) s[(base + 256 * q) % CB][(base + 256 * q) / CB] = v[q];
  }
  __syncthreads();
  // off-diagonal quadrant at (oi, ok): Y = T W(ok, ok), then -W(oi, oi) Y.
  // Every thread holds a 4 x 4 part of the 64 x 64 product (rows ti + 16 a,
  // columns tj + 16 b), so a step of k costs 8 shared-memory loads for 16
  // FMAs; one load per operand of each FMA took 35 us here, this takes 16.
  const int oi = lower ? BS : 0, ok = lower ? 0 : BS, ti = tid % 16, tj = tid / 16;
  T y[4][4];
#pragma unroll
  for (int pass = 0; pass < 2; pass++) {
    const T *L = &s[oi + ti][pass ? oi : ok], *R = &s[pass ? oi : ok][ok + tj];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int c = 0; c < 4; c++) y[a][c] = T(0);
#pragma unroll 4
    for (int k = 0; k < BS; k++) {
      T l[4], r[4];
#pragma unroll
      for (int a = 0; a < 4; a++) l[a] = L[16 * a * (CB + 1) + k];
#pragma unroll
      for (int c = 0; c < 4; c++) r[c] = R[k * (CB + 1) + 16 * c];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int c = 0; c < 4; c++) y[a][c] = fma(l[a], r[c], y[a][c]);
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int c = 0; c < 4; c++) s[oi + ti + 16 * a][ok + tj + 16 * c] = pass ? -y[a][c] : y[a][c];
    __syncthreads();
  }
  T *Wb = W128 + (long)b * CB * CB;
  for (int idx = tid; idx < CB * CB; idx += 256) Wb[idx] = s[idx % CB][idx / CB];
}

}  // namespace

size_t trsv_w_elems(int n) { return (size_t)cdiv(n, CB) * CB * CB + (size_t)cdiv(n, BS) * BS * BS; }

// Inverted 128 x 128 diagonal blocks of op(A)'s triangle, as trsv_w_dev takes
// them (W holds trsv_w_elems(n) elements: the 128 x 128 inverses, then the
// 64 x 64 ones they are assembled from).
template <typename T>
void trsv_inverse_dev(int uplo, int trans, int diag, int n, const T *A, long lda, T *W, cudaStream_t st) {
  if (n <= 0) return;
  const bool tr = trans != kNoTrans;
  const long tstr = tr ? lda : 1, tcol = tr ? 1 : lda;
  const int lower = (uplo == kLower) != tr;
  T *W64 = W + (size_t)cdiv(n, CB) * CB * CB;
  trinv_dev<T>(n, A, tstr, tcol, lower, diag == kUnit, W64, st);
  constexpr int smem = CB * (CB + 1) * (int)sizeof(T);
  static bool configured = false;
  if (!configured) {
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(trinv128_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  trinv128_kernel<T><<<cdiv(n, CB), 256, smem, st>>>(n, A, tstr, tcol, lower, W64, W);
  ATLB_CUDA_CHECK(cudaGetLastError());
}
template void trsv_inverse_dev<double>(int, int, int, int, const double *, long, double *, cudaStream_t);
template void trsv_inverse_dev<float>(int, int, int, int, const float *, long, float *, cudaStream_t);

// Solve op(A) X = B in place (Left side only): the inverted diagonal blocks
// once, then one launch per 16 (FP64) or 8 right-hand sides.
template <typename T>
void trsv_dev(int uplo, int trans, int diag, int n, int nrhs, const T *A, long lda, T *B, long ldb,
              cudaStream_t st) {
  if (n <= 0 || nrhs <= 0) return;
  T *W = (T *)scratch(kSlotTrsmW, sizeof(T) * trsv_w_elems(n));
  trsv_inverse_dev<T>(uplo, trans, diag, n, A, lda, W, st);
  constexpr int step = sizeof(T) == 8 ? 16 : 8;  // right-hand sides of one launch
  for (int c0 = 0; c0 < nrhs; c0 += step)
    trsv_w_dev<T>(uplo, trans, n, std::min(step, nrhs - c0), A, lda, W, B + (long)c0 * ldb, ldb, st);
}
template void trsv_dev<double>(int, int, int, int, int, const double *, long, double *, long, cudaStream_t);
template void trsv_dev<float>(int, int, int, int, int, const float *, long, float *, long, cudaStream_t);

// The same solve with the inverted diagonal blocks W already computed
// (trsv_inverse_dev): for repeated solves with one factor; nrhs <= 16 (FP64)
// or 8.
template <typename T>
void trsv_w_dev(int uplo, int trans, int n, int nrhs, const T *A, long lda, const T *W, T *B, long ldb,
                cudaStream_t st) {
  if (n <= 0 || nrhs <= 0) return;
  const bool tr = trans != kNoTrans;
  const long tstr = tr ? lda : 1, tcol = tr ? 1 : lda;  // effective T(i,k) = A[i*tstr + k*tcol]
  const int lower = (uplo == kLower) != tr;
  const int nb = cdiv(n, CB);
  // workspace: ticket counter, flags, and (FP32) the tagged copy
  // of x, 8 words per row
  const size_t nctl = (size_t)cdiv(nb + 64, 2) * 2, ntag = sizeof(T) == 4 ? (size_t)nb * CB * 8 : 0;
  int *ctl = (int *)scratch(kSlotTrsvCtl, sizeof(int) * nctl + sizeof(unsigned long long) * ntag);
  const int epoch = 1;
  int *counter = ctl, *flags = ctl + 64, *word = wait_word();
  unsigned long long *xt = (unsigned long long *)(ctl + nctl);
  ATLB_CUDA_CHECK(cudaMemsetAsync(ctl, 0, sizeof(int) * nctl + sizeof(unsigned long long) * ntag, st));
  // sW, sxd, sb, sacc (trsv_kernel's layout), for the largest NR
  constexpr int smem = (CB * (CB + 1) + (2 * CB + CB + NQ * CB) * 8) * (int)sizeof(T);
  if constexpr (sizeof(T) == 8) {
    if (nrhs > 1 || (n > 2 * CB && tstr != 1)) {
      constexpr int smem1 = (CB * (CB + 4) + 3 * CB * 12) * 8, smem2 = (CB * (CB + 4) + 3 * CB * 20) * 8;
      static bool configured_m = false;
      if (!configured_m) {
        ATLB_CUDA_CHECK(cudaFuncSetAttribute(trsv_mma_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem1));
        ATLB_CUDA_CHECK(cudaFuncSetAttribute(trsv_mma_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2));
        configured_m = true;
      }
      if (nrhs <= 8)
        trsv_mma_kernel<1><<<nb, TT, smem1, st>>>(n, nrhs, A, tstr, tcol, lower, W, B, ldb, counter, flags, epoch, word);
      else
        trsv_mma_kernel<2><<<nb, TT, smem2, st>>>(n, nrhs, A, tstr, tcol, lower, W, B, ldb, counter, flags, epoch, word);
      ATLB_CUDA_CHECK(cudaGetLastError());
      return;
    }
  }
  static bool configured = false;
  if (!configured) {
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(trsv_kernel<T, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if constexpr (sizeof(T) == 4) {
      ATLB_CUDA_CHECK(cudaFuncSetAttribute(trsv_kernel<T, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      ATLB_CUDA_CHECK(cudaFuncSetAttribute(trsv_kernel<T, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    }
    configured = true;
  }
  auto go = [&](auto kern) {
    kern<<<nb, TT, smem, st>>>(n, nrhs, A, tstr, tcol, lower, W, B, ldb, counter, flags, epoch, word, xt);
  };
  if constexpr (sizeof(T) == 8) go(trsv_kernel<T, 1>);
  else if (nrhs == 1) go(trsv_kernel<T, 1>);
  else if (nrhs <= 4) go(trsv_kernel<T, 4>);
  else go(trsv_kernel<T, 8>);
  ATLB_CUDA_CHECK(cudaGetLastError());
}
template void trsv_w_dev<double>(int, int, int, int, const double *, long, const double *, double *, long,
                                 cudaStream_t);
template void trsv_w_dev<float>(int, int, int, int, const float *, long, const float *, float *, long,
                                cudaStream_t);

}  // namespace atlb
