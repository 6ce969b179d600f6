// FP64 GEMM on the sm_100a FP64 tensor path (DMMA, mma.sync m8n8k4 f64).
//
// Replaces the amm micro-kernels + block copies of the reference GEMM driver
// (src/blas/ammm/ATL_ammm.c:12-364, ATL_iploops.c:19-181): instead of copying
// A/B into access-major blocks on the host, a 4-stage cp.async pipeline stages
// 128x16 tiles of op(A) and op(B) in shared memory in the layout their global
// memory already has (no transposing copy), and each of 8 warps accumulates a
// 64x32 block of C in registers with DMMA.  The same kernel computes one
// triangle of C for SYRK (tiles outside the triangle exit at once; elements
// outside it are not stored).
#include <algorithm>
#include <cstring>
#include <vector>
#include "common.cuh"
#include "kernels.h"

namespace atlb {
namespace {

constexpr int BM = 128, BN = 128, BK = 16, THREADS = 256, STAGES = 4, PAD = 4;

// Shared-memory layout of one operand tile of BO (outer) x BK.  "o" is the
// outer index (m for A, n for B), "k" the reduction index.  KC = the operand
// is k-contiguous in global memory (A transposed, B not transposed);
// otherwise o-contiguous.
template <bool KC, int BO> struct Lay;
template <int BO> struct Lay<false, BO> {
  static constexpr int LD = BO + PAD;  // 132 / 68 doubles (4 mod 16): conflict-free fragments
  static constexpr int SIZE = BK * LD;
  __device__ static __forceinline__ int at(int o, int k) { return k * LD + o; }
};
template <int BO> struct Lay<true, BO> {
  static constexpr int LD = BK + PAD;  // 20 doubles
  static constexpr int SIZE = BO * LD;
  __device__ static __forceinline__ int at(int o, int k) { return o * LD + k; }
};

// Issue the cp.async copies of one BO x BK tile (o0.., k0..) of an operand.
template <bool KC, int VEC, int BO, int NTHR = THREADS, int UNROLL = 16>
__device__ __forceinline__ void load_tile(double *s, const double *X, long ld, int o0, int k0,
                                          int O, int K, int tid) {
  using L = Lay<KC, BO>;
  constexpr int N16 = BO * BK / 2 / NTHR, N8 = BO * BK / NTHR;  // copies per thread
  if (!KC) {
    if (VEC == 2) {
#pragma unroll
      for (int i = 0; i < N16; i++) {
        int c = tid + NTHR * i, k = c / (BO / 2), o = (c % (BO / 2)) * 2;
        int go = o0 + o, gk = k0 + k;
        double *d = s + L::at(o, k);
        const double *g = X + go + (long)gk * ld;
        if (gk < K && go + 1 < O) cp_async16(d, g, true);
        else {
          bool p0 = gk < K && go < O;
          cp_async8(d, p0 ? g : X, p0);
          cp_async8(d + 1, X, false);
        }
      }
    } else {
#pragma unroll UNROLL
      for (int i = 0; i < N8; i++) {
        int c = tid + NTHR * i, k = c / BO, o = c % BO;
        int go = o0 + o, gk = k0 + k;
        bool p = gk < K && go < O;
        cp_async8(s + L::at(o, k), p ? X + go + (long)gk * ld : X, p);
      }
    }
  } else {
    if (VEC == 2) {
#pragma unroll
      for (int i = 0; i < N16; i++) {
        int c = tid + NTHR * i, o = c >> 3, k = (c & 7) * 2;
        int go = o0 + o, gk = k0 + k;
        double *d = s + L::at(o, k);
        const double *g = X + gk + (long)go * ld;
        if (go < O && gk + 1 < K) cp_async16(d, g, true);
        else {
          bool p0 = go < O && gk < K;
          cp_async8(d, p0 ? g : X, p0);
          cp_async8(d + 1, X, false);
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < N8; i++) {
        int c = tid + NTHR * i, o = c >> 4, k = c & 15;
        int go = o0 + o, gk = k0 + k;
        bool p = go < O && gk < K;
        cp_async8(s + L::at(o, k), p ? X + gk + (long)go * ld : X, p);
      }
    }
  }
}

// The same for 16-byte copies of tiles that lie wholly inside the operand, from a
// pointer to the thread's first element: no bounds to test, and the addresses of a
// thread's copies are a fixed stride apart.  Bounds and 64-bit addresses were most
// of the instructions of a short-K tile (a 128 x 64 tile with K = 128: 38,000 warp
// instructions, 4,096 of them products); with this and the untested epilogue
// 8192^2 x 128 goes from 25.8 to 28.3 TFLOP/s, 8192^3 from 34.7 to 35.7.  Eight-byte
// copies keep the tested form: twice the addresses left the registers short (1501 x
// 1203 x 999, A transposed: 160 -> 178 us).
template <bool KC, int BO> struct TileCopy {
  using L = Lay<KC, BO>;
  static constexpr int PER = (KC ? BK : BO) / 2;  // copies along the contiguous direction
  static constexpr int ROWS = THREADS / PER, N = BO * BK / 2 / THREADS;
  static __device__ __forceinline__ const double *first(const double *X, long ld, int o0, int tid) {
    const int c = tid % PER * 2, r = tid / PER;
    return KC ? X + c + (long)(o0 + r) * ld : X + o0 + c + (long)r * ld;
  }
  static __device__ __forceinline__ void go(double *s, const double *g, long ld, int tid) {
    double *d = s + tid / PER * L::LD + tid % PER * 2;
    const long step = ROWS * ld;
#pragma unroll
    for (int i = 0; i < N; i++) {
      cp_async16(d + i * ROWS * L::LD, g, true);
      g += step;
    }
  }
};

// Tile shapes.  BNT = 128: 128 x 128 tiles, 4 stages, one CTA per SM (the
// long-K GEMMs).  BNT = 64: 128 x 64 tiles, 3 stages, two CTAs per SM, so
// that one CTA's epilogue (the old C tile in and the new one out) overlaps
// the other's main loop -- the short-K trailing updates of the
// factorizations (K = 128..256), where a 128 x 128 tile spends a large part
// of its time in the epilogue.
template <int BNT> struct TileCfg {
  static constexpr int STG = BNT == 128 ? STAGES : 3;
  static constexpr int MINB = BNT == 128 ? 1 : 2;
  static constexpr int WARPS_N = BNT / 32, WARPS_M = 8 / WARPS_N;
  static constexpr int WMT = BM / WARPS_M, MI = WMT / 8;  // warp tile: WMT x 32 = MI x 4 fragments
  template <bool TA, bool TB>
  static constexpr int smem_doubles() { return STG * (Lay<TA, BM>::SIZE + Lay<!TB, BNT>::SIZE); }
};
// K up to this uses the 128 x 64 tiles: with bulk copies out the narrow tiles stay
// ahead for longer (8192^2 x 320 with C read back: 31.5 TFLOP/s wide, 33.5 narrow;
// x 512 33.0 and 34.1, 2048^2 x 512 28.3 and 28.7; at 640 on 2048^2 29.4 and 29.1)
constexpr int SMALL_K = 256, SMALL_K_BULK = 512;
constexpr int SMALL_TILE_K = 512;  // K up to this, with few tiles, uses 32 x 32 or 64 x 64 tiles
// the grouped (batched) GEMM's tile width: its problems are small (K <= 512,
// M, N from 16), where the narrower tile wastes less on padding and two CTAs
// per SM overlap their epilogues
constexpr int GROUPED_BN = 64;

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// One BM x BNT tile of C = alpha*op(A)*op(B) + beta*C (column-major) at
// (m0, n0).  tri: 0 full, 1 lower (store row >= col), 2 upper (row <= col).
// bulk: tiles that are stored whole leave by bulk copies (launch() says when).
template <bool TA, bool TB, int VEC, int BNT = BN>
__device__ __forceinline__ void dgemm_tile(int M, int N, int K, double alpha, const double *__restrict__ A,
                                           long lda, const double *__restrict__ B, long ldb, double beta,
                                           double *__restrict__ C, long ldc, int tri, int bulk, int m0, int n0,
                                           double *smem) {
  using CF = TileCfg<BNT>;
  constexpr int STG = CF::STG, MI = CF::MI;
  using LA = Lay<TA, BM>;     // A k-contiguous when transposed
  using LB = Lay<!TB, BNT>;   // B k-contiguous when not transposed
  double *sA = smem;
  double *sB = smem + STG * LA::SIZE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp % CF::WARPS_M) * CF::WMT, wn = (warp / CF::WARPS_M) * 32;

  double acc[MI][4][2];
#pragma unroll
  for (int i = 0; i < MI; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

  using CA = TileCopy<TA, BM>;
  using CB = TileCopy<!TB, BNT>;
  // eight-byte copies of the narrow tiles four at a time: with all eight addresses their
  // 128 registers spill (2500 x 2501 x 33, B transposed: 49.1 -> 47.0 us)
  constexpr int UN = BNT == 64 ? 4 : 16;
  const bool fullm = m0 + BM <= M, fulln = n0 + BNT <= N;
  const double *gA = CA::first(A, lda, m0, tid), *gB = CB::first(B, ldb, n0, tid);
  auto load_a = [&](int stage, int k0) {
    if (VEC == 2 && fullm && k0 + BK <= K) CA::go(sA + stage * LA::SIZE, gA + (TA ? k0 : k0 * lda), lda, tid);
    else load_tile<TA, VEC, BM, THREADS, UN>(sA + stage * LA::SIZE, A, lda, m0, k0, M, K, tid);
  };
  auto load_b = [&](int stage, int k0) {
    if (VEC == 2 && fulln && k0 + BK <= K) CB::go(sB + stage * LB::SIZE, gB + (TB ? k0 * ldb : k0), ldb, tid);
    else load_tile<!TB, VEC, BNT, THREADS, UN>(sB + stage * LB::SIZE, B, ldb, n0, k0, N, K, tid);
  };
  const int KT = (K + BK - 1) / BK;
#pragma unroll 1
  for (int s = 0; s < STG - 1; s++) {
    if (s < KT) {
      load_a(s, s * BK);
      load_b(s, s * BK);
    }
    cp_async_commit();
  }

  if (beta != 0.0 && !(VEC == 2 && bulk)) {  // the old C tile on its way to L2 while the products run
    for (int idx = tid; idx < BNT * (BM / 16); idx += THREADS) {
      const int r = m0 + idx % (BM / 16) * 16, c = n0 + idx / (BM / 16);
      if (r < M && c < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + r + (long)c * ldc));
    }
  }

  // The FP64 MMA unit is one per SM and a few warps keep it full, so what
  // costs is every warp being away from it at once: at a barrier, issuing
  // copies, waiting for the first fragments behind the barrier.  Fragments
  // are therefore loaded one k-step ahead, the barrier that opens the next k
  // tile stands before the last k-step's products (whose fragments are in
  // registers already), and the copies that refill the stage finished before
  // it are issued behind products too, A's and B's behind different k-steps: one
  // burst of both behind the last k-step needs more address registers than
  // there are (255 and spills without alignment; 1501 x 1203 x 999, A
  // transposed, 193 us, now 159).  8192^3: 31.5 -> 34.7 TFLOP/s (cuBLAS 35.5).
  const int fr = lane >> 2, fk = lane & 3;
  double a[2][MI], b[2][4];
  auto fragments = [&](int buf, const double *a_s, const double *b_s, int kk) {
#pragma unroll
    for (int i = 0; i < MI; i++) a[buf][i] = a_s[LA::at(wm + i * 8 + fr, kk + fk)];
#pragma unroll
    for (int j = 0; j < 4; j++) b[buf][j] = b_s[LB::at(wn + j * 8 + fr, kk + fk)];
  };
  cp_async_wait<STG - 2>();
  __syncthreads();
  fragments(0, sA, sB, 0);
  int stage = 0, refill = STG - 1;  // the stage read now, the one read before it
  for (int kt = 0; kt < KT; kt++) {
    const double *a_s = sA + stage * LA::SIZE, *b_s = sB + stage * LB::SIZE;
    stage = stage + 1 == STG ? 0 : stage + 1;
#pragma unroll
    for (int s = 0; s < BK / 4; s++) {
      if (s < BK / 4 - 1) {
        fragments((s + 1) & 1, a_s, b_s, 4 * (s + 1));
      } else {
        cp_async_commit();
        cp_async_wait<STG - 2>();
        __syncthreads();  // tile kt + 1 has landed, and nobody reads tile kt's stage any more
        if (kt + 1 < KT) fragments((s + 1) & 1, sA + stage * LA::SIZE, sB + stage * LB::SIZE, 0);
      }
#pragma unroll
      for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) dmma(acc[i][j], a[s & 1][i], b[s & 1][j]);
      if (kt + STG - 1 < KT) {
        const int k0 = (kt + STG - 1) * BK;
        if (s == 0) load_a(refill, k0);
        if (s == 1) load_b(refill, k0);
      }
    }
    refill = refill + 1 == STG ? 0 : refill + 1;
  }
  cp_async_wait<0>();

  // epilogue: C fragment row = lane>>2, cols = 2*(lane&3) + {0,1}.  With
  // beta != 0 the old C tile is first staged in shared memory (the pipeline
  // buffers are free now) by one burst of asynchronous copies, so its load
  // latency is paid once per tile rather than once per fragment row.
  auto ok = [&](int r, int c) {
    return r < M && c < N && !(tri == 1 && r < c) && !(tri == 2 && r > c);
  };
  // A tile that is stored whole needs no test per element.
  const bool whole = fullm && fulln && (tri == 0 || (tri == 1 ? m0 >= n0 + BNT - 1 : n0 >= m0 + BM - 1));
  constexpr int CLD = BM + 4;  // staged C: column-major, ld CLD (fits the pipeline buffers)
  static_assert(BNT * CLD <= STG * (Lay<false, BM>::SIZE + Lay<false, BNT>::SIZE), "C tile does not fit");
  double *sC = smem;
  // With beta = 0 or 1, a whole tile goes to shared memory and from there to
  // global memory by one bulk copy per column, which adds in L2 where beta = 1:
  // one rounding per element, as C + v has, and each element is added to once.
  // C is not read by the SM, and its load and store unit is free for the
  // fragments of the SM's other CTA: a warp's store of fragments touches 4
  // lines, and the 256 loads and 256 stores of a tile kept that unit for about
  // 4,000 cycles of the 16,400 that the products take with K = 128 (starting the
  // two CTAs half a tile apart, or loading the next tile during the epilogue,
  // gained nothing).  8192^2 x 128: 28.3 -> 31.6 TFLOP/s, x 64: 23.7 -> 28.8.
  if (VEC == 2 && whole && bulk) {
    constexpr int BLD = BM + 2;  // 2 mod 16: a fragment's 8 rows x 4 column pairs in distinct banks
    double *sc = sC + wm + fr + (wn + fk * 2) * BLD;
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < MI; i++) sc[i * 8 + (j * 8 + h) * BLD] = alpha * acc[i][j][h];
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid < BNT) {
      const uint32_t src = (uint32_t)__cvta_generic_to_shared(sC + tid * BLD);
      double *dst = C + m0 + (long)(n0 + tid) * ldc;
      if (beta == 0.0)
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src),
                     "n"(BM * 8) : "memory");
      else
        asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;" ::"l"(dst),
                     "r"(src), "n"(BM * 8) : "memory");
      asm volatile("cp.async.bulk.commit_group;\n cp.async.bulk.wait_group.read 0;" ::: "memory");
    }
    return;
  }
  if (beta != 0.0) {
    __syncthreads();  // every warp is done with the pipeline buffers
    const bool vec = VEC == 2 && (uintptr_t)C % 16 == 0 && ldc % 2 == 0;
    if (whole && vec) {
      constexpr int COLS = THREADS / (BM / 2);
      const int rr = tid % (BM / 2) * 2, cc = tid / (BM / 2);
      const double *g = C + m0 + rr + (long)(n0 + cc) * ldc;
      double *d = sC + rr + cc * CLD;
#pragma unroll 8
      for (int i = 0; i < BNT / COLS; i++) {
        cp_async16(d + i * COLS * CLD, g, true);
        g += COLS * ldc;
      }
    } else if (vec) {
#pragma unroll 4
      for (int idx = tid; idx < BM * BNT / 2; idx += THREADS) {
        const int rr = idx % (BM / 2) * 2, cc = idx / (BM / 2), r = m0 + rr, c = n0 + cc;
        const bool ok0 = ok(r, c), ok1 = ok(r + 1, c);
        const double *g = C + r + (long)c * ldc;
        double *d = sC + rr + cc * CLD;
        if (ok0 && ok1) cp_async16(d, g, true);
        else if (ok0) cp_async8(d, g, true);
        else if (ok1) cp_async8(d + 1, g + 1, true);
      }
    } else {
      for (int idx = tid; idx < BM * BNT; idx += THREADS) {
        const int rr = idx % BM, cc = idx / BM, r = m0 + rr, c = n0 + cc;
        if (ok(r, c)) cp_async8(sC + rr + cc * CLD, C + r + (long)c * ldc, true);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
  }
  if (whole) {
    const double *sc = sC + wm + fr + (wn + fk * 2) * CLD;
    double *g = C + m0 + wm + fr + (long)(n0 + wn + fk * 2) * ldc;
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        double *gc = g + (j * 8 + h) * ldc;
#pragma unroll
        for (int i = 0; i < MI; i++) {
          double v = alpha * acc[i][j][h];
          if (beta != 0.0) v = fma(beta, sc[i * 8 + (j * 8 + h) * CLD], v);
          gc[i * 8] = v;
        }
      }
    return;
  }
#pragma unroll
  for (int i = 0; i < MI; i++) {
    const int rr = wm + i * 8 + fr, r = m0 + rr;
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int cc = wn + j * 8 + fk * 2 + h, c = n0 + cc;
        if (!ok(r, c)) continue;
        double v = alpha * acc[i][j][h];
        if (beta != 0.0) v = fma(beta, sC[rr + cc * CLD], v);
        C[r + (long)c * ldc] = v;
      }
  }
}

template <bool TA, bool TB, int VEC, int BNT>
__global__ void __launch_bounds__(THREADS, TileCfg<BNT>::MINB)
dgemm_dmma_kernel(int M, int N, int K, double alpha, const double *__restrict__ A, long lda,
                  const double *__restrict__ B, long ldb, double beta, double *__restrict__ C,
                  long ldc, int tri, int bulk, int G) {
  extern __shared__ __align__(16) double smem[];
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BNT - 1) / BNT;
  // grouped rasterisation: G tile-rows share B panels in L2
  const int bid = blockIdx.x;
  const int per_group = G * tiles_n, group = bid / per_group;
  const int first_m = group * G, gsz = min(tiles_m - first_m, G);
  const int tm = first_m + (bid % per_group) % gsz, tn = (bid % per_group) / gsz;
  const int m0 = tm * BM, n0 = tn * BNT;
  if (tri == 1 && m0 + BM - 1 < n0) return;
  if (tri == 2 && m0 > n0 + BNT - 1) return;
  dgemm_tile<TA, TB, VEC, BNT>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, tri, bulk, m0, n0, smem);
}

// GEMMs whose output has too few 128 x 128 tiles for the SMs and whose K is
// short (the small updates inside the factorizations, a user's small
// products): BT x BT tiles (32, or 64 for many of them without alignment), four
// warps, old C fetched into registers before the main loop.  Split K
// needs a second launch and a round trip of the partials through memory,
// which is most of the time of such a product.  Against split K (device time,
// launches included): 128^3 14.4 -> 7.5 us, 96 x 80 x 112 16.2 -> 8.9,
// 1000 x 128 x 128 14.5 -> 8.7, 8000 x 128 x 128 28.2 -> 18.4,
// 1000 x 1000 x 500 63.6 -> 49.9.
constexpr int SM_THREADS = 128, SM_STAGES = 3;
template <bool TA, bool TB, int BT>
constexpr int small_smem() { return SM_STAGES * (Lay<TA, BT>::SIZE + Lay<!TB, BT>::SIZE) * (int)sizeof(double); }

template <bool TA, bool TB, int VEC, int BT>
__global__ void __launch_bounds__(SM_THREADS)
dgemm_small_kernel(int M, int N, int K, double alpha, const double *__restrict__ A, long lda,
                   const double *__restrict__ B, long ldb, double beta, double *__restrict__ C,
                   long ldc, int tri) {
  extern __shared__ __align__(16) double smem[];
  using LA = Lay<TA, BT>;
  using LB = Lay<!TB, BT>;
  constexpr int WT = BT / 2, MI = WT / 8;  // a warp's part: WT x WT
  double *sA = smem, *sB = smem + SM_STAGES * LA::SIZE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tiles_m = (M + BT - 1) / BT;
  const int m0 = (blockIdx.x % tiles_m) * BT, n0 = (blockIdx.x / tiles_m) * BT;
  if (tri == 1 && m0 + BT - 1 < n0) return;
  if (tri == 2 && m0 > n0 + BT - 1) return;
  const int fr = lane >> 2, fk = lane & 3, wm = (warp & 1) * WT, wn = (warp >> 1) * WT;
  const int KT = (K + BK - 1) / BK;
  auto load = [&](int kt) {
    if (kt < KT) {
      load_tile<TA, VEC, BT, SM_THREADS>(sA + kt % SM_STAGES * LA::SIZE, A, lda, m0, kt * BK, M, K, tid);
      load_tile<!TB, VEC, BT, SM_THREADS>(sB + kt % SM_STAGES * LB::SIZE, B, ldb, n0, kt * BK, N, K, tid);
    }
    cp_async_commit();
  };
#pragma unroll 1
  for (int s = 0; s < SM_STAGES - 1; s++) load(s);
  auto ok = [&](int r, int c) {
    return r < M && c < N && !(tri == 1 && r < c) && !(tri == 2 && r > c);
  };
  double acc[MI][MI][2], old[MI][MI][2];
#pragma unroll
  for (int i = 0; i < MI; i++)
#pragma unroll
    for (int j = 0; j < MI; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = m0 + wm + i * 8 + fr, c = n0 + wn + j * 8 + fk * 2 + h;
        acc[i][j][h] = 0.0;
        old[i][j][h] = beta != 0.0 && ok(r, c) ? C[r + (long)c * ldc] : 0.0;
      }
#pragma unroll 1
  for (int kt = 0; kt < KT; kt++) {
    cp_async_wait<SM_STAGES - 2>();
    __syncthreads();
    load(kt + SM_STAGES - 1);
    const double *a_s = sA + kt % SM_STAGES * LA::SIZE, *b_s = sB + kt % SM_STAGES * LB::SIZE;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      double a[MI], b[MI];
#pragma unroll
      for (int i = 0; i < MI; i++) {
        a[i] = a_s[LA::at(wm + i * 8 + fr, kk + fk)];
        b[i] = b_s[LB::at(wn + i * 8 + fr, kk + fk)];
      }
#pragma unroll
      for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < MI; j++) dmma(acc[i][j], a[i], b[j]);
    }
  }
  cp_async_wait<0>();
#pragma unroll
  for (int i = 0; i < MI; i++)
#pragma unroll
    for (int j = 0; j < MI; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = m0 + wm + i * 8 + fr, c = n0 + wn + j * 8 + fk * 2 + h;
        if (!ok(r, c)) continue;
        double v = alpha * acc[i][j][h];
        if (beta != 0.0) v = fma(beta, old[i][j][h], v);
        C[r + (long)c * ldc] = v;
      }
}

// The same GEMM on a capped number of CTAs, each walking tiles t, t + grid,
// ... (same rasterisation): leaves SMs free for work on another stream
// (the factorizations' look-ahead panels).
template <bool TA, bool TB, int VEC>
__global__ void __launch_bounds__(THREADS, 1)
dgemm_capped_kernel(int M, int N, int K, double alpha, const double *__restrict__ A, long lda,
                    const double *__restrict__ B, long ldb, double beta, double *__restrict__ C,
                    long ldc, int tri, int bulk, int G) {
  extern __shared__ __align__(16) double smem[];
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN, tiles = tiles_m * tiles_n;
  for (int bid = blockIdx.x; bid < tiles; bid += gridDim.x) {
    const int per_group = G * tiles_n, group = bid / per_group;
    const int first_m = group * G, gsz = min(tiles_m - first_m, G);
    const int tm = first_m + (bid % per_group) % gsz, tn = (bid % per_group) / gsz;
    const int m0 = tm * BM, n0 = tn * BN;
    if (tri == 1 && m0 + BM - 1 < n0) continue;
    if (tri == 2 && m0 > n0 + BN - 1) continue;
    dgemm_tile<TA, TB, VEC>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, tri, bulk, m0, n0, smem);
    __syncthreads();  // shared memory is reused by the next tile
  }
}

// Grouped (batched, uneven) GEMM: a persistent grid walks the 128x128 tiles
// of all problems; tile t belongs to problem order[p] where tile_start[p] <= t
// < tile_start[p+1] (problems sorted by decreasing size on the host).
template <bool TA, bool TB, int VEC, int BNT>
__global__ void __launch_bounds__(THREADS, TileCfg<BNT>::MINB)
dgemm_grouped_kernel(const GemmProb *__restrict__ probs, const int *__restrict__ order,
                     const int *__restrict__ tile_start, int count, int *__restrict__ next) {
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_t;
  const int total = tile_start[count];
  while (true) {
    if (threadIdx.x == 0) s_t = atomicAdd(next, 1);
    __syncthreads();
    const int t = s_t;
    if (t >= total) return;
    int lo = 0, hi = count - 1;  // last p with tile_start[p] <= t
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tile_start[mid] <= t) lo = mid; else hi = mid - 1;
    }
    const GemmProb pr = probs[order[lo]];
    const int local = t - tile_start[lo], tiles_n = (pr.N + BNT - 1) / BNT;
    const int m0 = (local / tiles_n) * BM, n0 = (local % tiles_n) * BNT;
    dgemm_tile<TA, TB, VEC, BNT>(pr.M, pr.N, pr.K, pr.alpha, pr.A, pr.lda, pr.B, pr.ldb, pr.beta, pr.C,
                                 pr.ldc, 0, 0, m0, n0, smem);
    __syncthreads();  // shared memory is reused by the next tile
  }
}

// Split-K for GEMMs with too few output tiles to fill the GPU (the small
// updates inside the factorizations): CTA (tile, s) multiplies over the s-th
// K range into its own dense partial P_s (ld = M); a second kernel sums the
// partials in a fixed order (deterministic) and applies alpha, beta and tri.
template <bool TA, bool TB, int VEC>
__global__ void __launch_bounds__(THREADS, 1)
dgemm_splitk_kernel(int M, int N, int K, int kc, const double *__restrict__ A, long lda,
                    const double *__restrict__ B, long ldb, double *__restrict__ P) {
  extern __shared__ __align__(16) double smem[];
  const int tiles_m = (M + BM - 1) / BM;
  const int tm = blockIdx.x % tiles_m, tn = blockIdx.x / tiles_m, s = blockIdx.y;
  const int k0 = s * kc, kl = min(kc, K - k0);
  const double *As = TA ? A + k0 : A + (long)k0 * lda;
  const double *Bs = TB ? B + (long)k0 * ldb : B + k0;
  dgemm_tile<TA, TB, VEC>(M, N, kl, 1.0, As, lda, Bs, ldb, 0.0, P + (long)s * M * N, M, 0, M % 2 == 0, tm * BM,
                          tn * BN, smem);
}

__global__ void splitk_reduce_kernel(int M, int N, int S, double alpha, const double *__restrict__ P,
                                     double beta, double *__restrict__ C, long ldc, int tri) {
  const long total = (long)M * N, mn = total;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
       idx += (long)gridDim.x * blockDim.x) {
    const int r = (int)(idx % M), c = (int)(idx / M);
    if (tri == 1 && r < c) continue;
    if (tri == 2 && r > c) continue;
    double acc = 0.0;
    for (int s = 0; s < S; s++) acc += P[idx + s * mn];
    double *p = C + r + (long)c * ldc;
    double v = alpha * acc;
    if (beta != 0.0) v = fma(beta, *p, v);
    *p = v;
  }
}

__global__ void scale_kernel(int M, int N, double beta, double *C, long ldc, int tri) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  long total = (long)M * N;
  for (; idx < total; idx += (long)gridDim.x * blockDim.x) {
    int r = (int)(idx % M), c = (int)(idx / M);
    if (tri == 1 && r < c) continue;
    if (tri == 2 && r > c) continue;
    double *p = C + r + (long)c * ldc;
    *p = (beta == 0.0) ? 0.0 : beta * *p;
  }
}

// Slices for a split-K GEMM of `tiles` output tiles (too few for the SMs):
// the smallest count, slices of at least 2 BK, whose CTAs (tiles x slices)
// fill their waves of nsm within 3 % of the best count -- e.g. 63 tiles take
// 7 slices (441 CTAs in 3 full waves), not 3 (189 CTAs, a second wave of 41).
int splitk_count(int tiles, int K, int nsm) {
  const int smax = std::max(1, std::min(K / (2 * BK), 4 * nsm));
  auto fill = [&](int s) {
    const long c = (long)tiles * s;
    return (double)c / ((double)cdiv(c, (long)nsm) * nsm);
  };
  double best = 0.0;
  for (int s = 1; s <= smax; s++) best = std::max(best, fill(s));
  for (int s = 1; s <= smax; s++)
    if (fill(s) >= 0.97 * best) return s;
  return 1;
}

}  // namespace

// Memory of the current device: the bulk copies' additions take place in its L2.
// Host, managed and other devices' memory keeps the loads and stores.  (0.3 us on
// the host, and no state: an address says nothing about the next call's, so a
// graph of launches that write a caller's matrix has the answer in its key.)
bool own_memory(const void *p) {
  cudaPointerAttributes a;
  int dev = -1;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice && a.device == dev;
}

namespace {

template <bool TA, bool TB, int VEC>
void launch(int M, int N, int K, double alpha, const double *A, long lda, const double *B,
            long ldb, double beta, double *C, long ldc, int tri, cudaStream_t st) {
  constexpr int smem = TileCfg<BN>::template smem_doubles<TA, TB>() * (int)sizeof(double);
  constexpr int smem_s = TileCfg<64>::template smem_doubles<TA, TB>() * (int)sizeof(double);
  static bool configured = false;
  if (!configured) {
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(dgemm_dmma_kernel<TA, TB, VEC, BN>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(dgemm_dmma_kernel<TA, TB, VEC, 64>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem_s));
    // the largest shared-memory carveout, so that two of these CTAs fit on an SM
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(dgemm_dmma_kernel<TA, TB, VEC, 64>,
                                         cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    configured = true;
  }
  int tiles = cdiv(M, BM) * cdiv(N, BN);
  const int nsm = num_sms();
  // Too few tiles for the 148 SMs: smaller tiles while K is short, else split K
  // (partials + reduction).  Where an SM has one 32 x 32 tile or less, that tile's
  // serial K loop becomes the longer towards K = 512, without alignment from 450 on
  // (200 x 200 with C read back, split and small: K = 400 16.6 and 12.5 us, 450 16.6 and
  // 14.5, 512 14.6 and 14.5, A transposed 14.6 and 16.6; unaligned 16.6 and 14.6, 16.6
  // and 16.6, 14.6 and 17.4).  With more tiles than SMs the small ones are ahead at 512
  // too (500 x 500 20.7 and 17.6, 800 x 800 43.3 and 35.0).
  const long t32 = (long)cdiv(M, 32) * cdiv(N, 32), t64 = (long)cdiv(M, 64) * cdiv(N, 64);
  const bool can_split = tune(kTuneSplitK) && !no_alloc_active();
  const int most_k = !can_split || t32 > nsm ? SMALL_TILE_K : VEC == 2 ? 480 : 400;
  if (tiles * 2 <= nsm && K <= most_k) {
    auto go = [&](auto kern, int bt, int bytes, bool &set) {
      if (!set) {
        ATLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        ATLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        set = true;
      }
      kern<<<cdiv(M, bt) * cdiv(N, bt), SM_THREADS, bytes, st>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, tri);
      ATLB_CUDA_CHECK(cudaGetLastError());
    };
    // 64 x 64 tiles cost four of 32 x 32 each and leave more of the last wave idle
    // (800 x 800 x 512, 169 tiles: 47.4 us, 32 x 32 35.1).  With 16-byte copies the small
    // ones are ahead throughout (1000^2 x 512 47.2 and 51.4); with 8-byte copies, which
    // cost them 1.25 times as much, where the waves say so (1000^2 x 512 59.6 and 53.5,
    // 900^2 47.3 and 53.4).
    if constexpr (VEC == 1) {
      if (t64 >= nsm && 16 * cdiv(t64, nsm) <= 5 * cdiv(t32, nsm)) {
        static bool set64 = false;
        go(dgemm_small_kernel<TA, TB, VEC, 64>, 64, small_smem<TA, TB, 64>(), set64);
        return;
      }
    }
    static bool set32 = false;
    go(dgemm_small_kernel<TA, TB, VEC, 32>, 32, small_smem<TA, TB, 32>(), set32);
    return;
  }
  int S = 1;
  if (can_split && tiles * 2 <= nsm && K >= 4 * BK) S = splitk_count(tiles, K, nsm);
  if (S > 1) {
    const int kc = cdiv(cdiv(K, S), BK) * BK;
    S = cdiv(K, kc);
    double *P = (double *)scratch(kSlotGemmSplit, sizeof(double) * (size_t)S * M * N);
    if (P) {
      static bool configured_s = false;
      if (!configured_s) {
        ATLB_CUDA_CHECK(cudaFuncSetAttribute(dgemm_splitk_kernel<TA, TB, VEC>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured_s = true;
      }
      dgemm_splitk_kernel<TA, TB, VEC><<<dim3(tiles, S), THREADS, smem, st>>>(M, N, K, kc, A, lda, B, ldb, P);
      const long total = (long)M * N;
      splitk_reduce_kernel<<<(int)std::min<long>((total + 255) / 256, 148L * 8), 256, 0, st>>>(
          M, N, S, alpha, P, beta, C, ldc, tri);
      ATLB_CUDA_CHECK(cudaGetLastError());
      return;
    }
  }
  // bulk copies out of shared memory want 16-byte alignment
  const int bulk = (beta == 0.0 || beta == 1.0) && (uintptr_t)C % 16 == 0 && ldc % 2 == 0 && own_memory(C);
  const int cap = gemm_cta_cap();
  if (cap > 0 && tiles > cap) {
    static bool configured_c = false;
    if (!configured_c) {
      ATLB_CUDA_CHECK(cudaFuncSetAttribute(dgemm_capped_kernel<TA, TB, VEC>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      configured_c = true;
    }
    dgemm_capped_kernel<TA, TB, VEC><<<cap, THREADS, smem, st>>>(M, N, K, alpha, A, lda, B, ldb, beta, C,
                                                                 ldc, tri, bulk, tune(kTuneGemmGroup));
    ATLB_CUDA_CHECK(cudaGetLastError());
    return;
  }
  // 128 x 64 tiles with long K too where they leave less of the last wave idle:
  // an SM computes two of them in the time of one 128 x 128 tile and 8 % (900 x
  // 1500 x 3000, as many waves both ways: 430 and 466 us), so they pay from
  // there (1700 x 1700 x 700, 196 tiles in 2 waves or 378 in 3 halves: 229 and
  // 183 us).  Not where a triangle is masked, whose tiles this does not count,
  // or a cap leaves SMs to another stream.
  const int tiles_n64 = cdiv(M, BM) * cdiv(N, 64);
  const bool finer = tri == 0 && cap == 0 && 27 * cdiv(tiles_n64, nsm) < 50 * cdiv(tiles, nsm);
  if (K <= SMALL_K || (VEC == 2 && bulk && K <= SMALL_K_BULK && tiles > nsm) || finer) {
    dgemm_dmma_kernel<TA, TB, VEC, 64><<<tiles_n64, THREADS, smem_s, st>>>(
        M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, tri, bulk, tune(kTuneGemmGroup));
  } else {
    dgemm_dmma_kernel<TA, TB, VEC, BN><<<tiles, THREADS, smem, st>>>(M, N, K, alpha, A, lda, B, ldb,
                                                                     beta, C, ldc, tri, bulk, tune(kTuneGemmGroup));
  }
  ATLB_CUDA_CHECK(cudaGetLastError());
}

inline bool al16(const void *p, long ld) { return ((uintptr_t)p % 16 == 0) && (ld % 2 == 0); }

}  // namespace

void dgemm_dev(int ta, int tb, int M, int N, int K, double alpha, const double *A, long lda,
               const double *B, long ldb, double beta, double *C, long ldc, cudaStream_t st,
               int tri) {
  if (M <= 0 || N <= 0) return;
  if (K <= 0 || alpha == 0.0) {
    if (beta == 1.0) return;
    long total = (long)M * N;
    int blocks = (int)std::min<long>((total + 255) / 256, 148L * 16);
    scale_kernel<<<blocks, 256, 0, st>>>(M, N, beta, C, ldc, tri);
    ATLB_CUDA_CHECK(cudaGetLastError());
    return;
  }
  const bool tA = ta != kNoTrans, tB = tb != kNoTrans;
  const bool v2 = al16(A, lda) && al16(B, ldb);
#define ATLB_DG(TA_, TB_)                                                                 \
  if (v2) launch<TA_, TB_, 2>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, tri, st);    \
  else launch<TA_, TB_, 1>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, tri, st);
  if (!tA && !tB) { ATLB_DG(false, false) }
  else if (!tA && tB) { ATLB_DG(false, true) }
  else if (tA && !tB) { ATLB_DG(true, false) }
  else { ATLB_DG(true, true) }
#undef ATLB_DG
}

namespace {
template <bool TA, bool TB, int VEC>
void launch_grouped(const GemmProb *probs, const int *order, const int *tile_start, int count,
                    int *next, cudaStream_t st) {
  constexpr int smem = TileCfg<GROUPED_BN>::template smem_doubles<TA, TB>() * (int)sizeof(double);
  static bool configured = false;
  if (!configured) {
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(dgemm_grouped_kernel<TA, TB, VEC, GROUPED_BN>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    ATLB_CUDA_CHECK(cudaFuncSetAttribute(dgemm_grouped_kernel<TA, TB, VEC, GROUPED_BN>,
                                         cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    configured = true;
  }
  dgemm_grouped_kernel<TA, TB, VEC, GROUPED_BN><<<num_sms() * TileCfg<GROUPED_BN>::MINB, THREADS, smem, st>>>(
      probs, order, tile_start, count, next);
  ATLB_CUDA_CHECK(cudaGetLastError());
}

}  // namespace

void dgemm_grouped_dev(int ta, int tb, const GemmProb *hp, int count, cudaStream_t st) {
  if (count <= 0) return;
  std::vector<int> order(count);
  for (int i = 0; i < count; i++) order[i] = i;
  auto work = [&](int i) { return (long)hp[i].M * hp[i].N * hp[i].K; };
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return work(a) > work(b); });
  std::vector<int> ts(count + 1, 0);
  bool v2 = true;
  for (int i = 0; i < count; i++) {
    const GemmProb &p = hp[order[i]];
    ts[i + 1] = ts[i] + ((p.M > 0 && p.N > 0) ? cdiv(p.M, BM) * cdiv(p.N, GROUPED_BN) : 0);
    v2 = v2 && al16(p.A, p.lda) && al16(p.B, p.ldb);
  }
  const size_t bytes = sizeof(GemmProb) * count + sizeof(int) * (2 * count + 1 + 16);
  unsigned char *d = (unsigned char *)scratch(kSlotBatch3, bytes);
  unsigned char *h = (unsigned char *)pinned(kSlotBatch3, bytes);
  memcpy(h, hp, sizeof(GemmProb) * count);
  memcpy(h + sizeof(GemmProb) * count, order.data(), sizeof(int) * count);
  memcpy(h + sizeof(GemmProb) * count + sizeof(int) * count, ts.data(), sizeof(int) * (count + 1));
  memset(h + sizeof(GemmProb) * count + sizeof(int) * (2 * count + 1), 0, sizeof(int) * 16);
  ATLB_CUDA_CHECK(cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st));
  const GemmProb *dp = (const GemmProb *)d;
  const int *dord = (const int *)(d + sizeof(GemmProb) * count);
  const int *dts = dord + count;
  int *next = (int *)(dts + count + 1);
  const bool tA = ta != kNoTrans, tB = tb != kNoTrans;
#define ATLB_GG(TA_, TB_)                                                     \
  if (v2) launch_grouped<TA_, TB_, 2>(dp, dord, dts, count, next, st);       \
  else launch_grouped<TA_, TB_, 1>(dp, dord, dts, count, next, st);
  if (!tA && !tB) { ATLB_GG(false, false) }
  else if (!tA && tB) { ATLB_GG(false, true) }
  else if (tA && !tB) { ATLB_GG(true, false) }
  else { ATLB_GG(true, true) }
#undef ATLB_GG
  // the host staging buffer must outlive the copy: wait for it here
  ATLB_CUDA_CHECK(cudaStreamSynchronize(st));
}

}  // namespace atlb
