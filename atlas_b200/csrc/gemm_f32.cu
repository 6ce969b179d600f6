// FP32 GEMM on the FP32 FMA pipes (cblas_sgemm and the FP32-exact factor
// mode of the mixed-precision solvers).  128x128x16 CTA tile, 128 threads,
// 8x16 outputs per thread (64x64 and 4x8 for few tiles); op(A) and op(B) tiles are staged in shared memory
// k-major (m / n contiguous) by a 3-stage cp.async pipeline, whatever their
// global layout, so the inner loop reads 128-bit vectors.  An output of few
// tiles with a long K (the Cholesky's diagonal-block updates) is split along
// K over gridDim.y: each slice writes its partial product to a workspace and
// one pass sums the slices into C.
// Reference semantics: src/blas/reference/level3/ATL_srefgemm.c.
#include <cstdint>
#include <type_traits>
#include "common.cuh"
#include "kernels.h"

namespace atlb {
namespace {

constexpr int BT = 128, BK = 16, THREADS = 128, STAGES = 3;
template <int T> constexpr int kLds = T + 4;
template <int T> constexpr int kSmem = 2 * STAGES * BK * kLds<T> * (int)sizeof(float);

// One T x 16 operand tile into shared memory, k-major (o contiguous).
// Operand element (o, k): TRANS_O ? X[k + o*ld] : X[o + k*ld].  VEC: o is
// contiguous in global memory and every column starts on 16 bytes, so whole
// 16-byte pieces are copied; otherwise 4 bytes at a time.
template <int T, bool TRANS_O, bool VEC>
__device__ __forceinline__ void load_tile(float *s, const float *X, long ld, int o0, int k0,
                                          int O, int K, int tid) {
  constexpr int LDS = kLds<T>;
  if (VEC && !TRANS_O) {
#pragma unroll
    for (int i = 0; i < T * BK / 4 / THREADS; i++) {
      const int c = tid + THREADS * i, o = c % (T / 4) * 4, k = c / (T / 4);
      const int go = o0 + o, gk = k0 + k;
      const float *g = X + go + (long)gk * ld;
      float *d = s + k * LDS + o;
      if (gk < K && go + 3 < O) cp_async16(d, g, true);
      else {
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const bool p = gk < K && go + e < O;
          cp_async4(d + e, p ? g + e : X, p);
        }
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < T * BK / THREADS; i++) {
      const int c = tid + THREADS * i;
      int o, k;
      if (!TRANS_O) { o = c % T; k = c / T; }   // o fastest: coalesced along o
      else { k = c & 15; o = c >> 4; }             // k fastest: coalesced along k
      const int go = o0 + o, gk = k0 + k;
      const bool p = go < O && gk < K;
      const float *g = TRANS_O ? X + gk + (long)go * ld : X + go + (long)gk * ld;
      cp_async4(s + k * LDS + o, p ? g : X, p);
    }
  }
}

// two FP32 fused multiply-adds in one instruction (each rounded as fmaf)
__device__ __forceinline__ void fma2(unsigned long long &c, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long swap2(unsigned long long x) {
  unsigned long long r;
  asm("{\n .reg .b32 lo, hi;\n mov.b64 {lo, hi}, %1;\n mov.b64 %0, {hi, lo};\n}" : "=l"(r) : "l"(x));
  return r;
}

// What bounds it: the FP32 pipes (74 TFLOP/s at 1965 MHz), so shared memory
// and the instructions issued must fit beside them.  A thread holds 8 x 16
// outputs: a k-step then costs a warp 24 shared-memory passes for 32 cycles of
// FMAs (with 8 x 8 outputs it was 16 for 16, and shared memory was the bound).
// Products go two to an instruction (fma.rn.f32x2): a pair of rows times a pair
// of columns, then the swapped pair of rows times the same, two moves a pair of
// rows.  4096^3: 3.17 ms with 8 x 8 outputs and single products, 2.76 ms
// now.
//
// Outputs of few 128 x 128 tiles take 64 x 64 ones (T = 64, 4 x 8 outputs a
// thread): four times the CTAs, and four warps' latency per tile a quarter as
// long.  With C read back, 128 x 128 tiles of 8 x 8 outputs and these: 128^3 23.1 and
// 9.0 us, 2000 x 128 x 128 26.9 and 10.7, 1000^3 140 and 75.  The line is at three
// small tiles an SM (111 large ones): with four, an SM is no sooner done than with
// one large tile.  Time with large tiles over that with small ones, K = 1000, A and B
// as they are / A transposed: 1.19 / 1.05 at 100 and 110 tiles, 0.91 / 0.81 at 121 to 144.
// Up to K = 128, where a tile's start and end count most, the small ones stay ahead
// to the last (121 tiles, K = 32 1.21 / 1.00, 128 1.00 / 0.91, unaligned 1.34 and 1.21).
template <int T, bool TA, bool TB, bool VA, bool VB>
__global__ void __launch_bounds__(THREADS, 2)
sgemm_simt_kernel(int M, int N, int K, float alpha, const float *__restrict__ A, long lda,
                  const float *__restrict__ B, long ldb, float beta, float *__restrict__ C,
                  long ldc, int tri, int kc, float *__restrict__ W) {
  if (gridDim.y > 1) {  // K slice blockIdx.y: its partial product, unscaled, into W's slice (ld M)
    const int k0 = blockIdx.y * kc;
    A += TA ? (long)k0 : (long)k0 * lda;
    B += TB ? (long)k0 * ldb : (long)k0;
    K = min(kc, K - k0);
    C = W + (long)blockIdx.y * M * N;
    ldc = M;
    alpha = 1.f;
    beta = 0.f;
  }
  constexpr int BM = T, BN = T, LDS = kLds<T>, H = T / 64;  // a warp's part: 32 H x 32 H
  extern __shared__ __align__(16) float sgemm_smem[];
  float *sA = sgemm_smem, *sB = sgemm_smem + STAGES * BK * LDS;
  const int tiles_m = (M + BM - 1) / BM, tiles_n = (N + BN - 1) / BN;
  const int bid = blockIdx.x, G = 8;
  const int per_group = G * tiles_n, group = bid / per_group;
  const int first_m = group * G, gsz = min(tiles_m - first_m, G);
  const int tm = first_m + (bid % per_group) % gsz, tn = (bid % per_group) / gsz;
  const int m0 = tm * BM, n0 = tn * BN;
  if (tri == 1 && m0 + BM - 1 < n0) return;
  if (tri == 2 && m0 > n0 + BN - 1) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this thread's rows rm + 32 h + 0..3 (h < H), columns cn + 16 q + 0..3 (q < 2 H)
  const int rm = (warp & 1) * 32 * H + (lane & 7) * 4, cn = (warp >> 1) * 32 * H + (lane >> 3) * 4;

  // row pair i x column pair j: acc[0] holds (row 0, col 0) and (row 1, col 1),
  // acc[1] (row 1, col 0) and (row 0, col 1)
  unsigned long long acc[2][2 * H][4 * H];
#pragma unroll
  for (int i = 0; i < 2 * H; i++)
#pragma unroll
    for (int j = 0; j < 4 * H; j++) acc[0][i][j] = acc[1][i][j] = 0ull;

  const int KT = (K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < STAGES - 1; s++) {
    if (s < KT) {
      load_tile<T, TA, VA>(sA + s * BK * LDS, A, lda, m0, s * BK, M, K, tid);
      load_tile<T, !TB, VB>(sB + s * BK * LDS, B, ldb, n0, s * BK, N, K, tid);
    }
    cp_async_commit();
  }
  for (int kt = 0; kt < KT; kt++) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    {
      const int nk = kt + STAGES - 1;
      if (nk < KT) {
        load_tile<T, TA, VA>(sA + nk % STAGES * BK * LDS, A, lda, m0, nk * BK, M, K, tid);
        load_tile<T, !TB, VB>(sB + nk % STAGES * BK * LDS, B, ldb, n0, nk * BK, N, K, tid);
      }
      cp_async_commit();
    }
    const float *as = sA + kt % STAGES * BK * LDS + rm, *bs = sB + kt % STAGES * BK * LDS + cn;
#pragma unroll
    for (int k = 0; k < BK; k++) {
      unsigned long long a[2 * H], b[4 * H], x[2 * H];
#pragma unroll
      for (int h = 0; h < H; h++) {
        const ulonglong2 ah = *reinterpret_cast<const ulonglong2 *>(as + k * LDS + 32 * h);
        a[2 * h] = ah.x;
        a[2 * h + 1] = ah.y;
      }
#pragma unroll
      for (int q = 0; q < 2 * H; q++) {
        const ulonglong2 bq = *reinterpret_cast<const ulonglong2 *>(bs + k * LDS + 16 * q);
        b[2 * q] = bq.x;
        b[2 * q + 1] = bq.y;
        x[q] = swap2(a[q]);
      }
#pragma unroll
      for (int j = 0; j < 4 * H; j++)
#pragma unroll
        for (int i = 0; i < 2 * H; i++) {
          fma2(acc[0][i][j], a[i], b[j]);
          fma2(acc[1][i][j], x[i], b[j]);
        }
    }
  }
  cp_async_wait<0>();
  // epilogue: a row quad of one column is contiguous in C.  Old C values are
  // loaded eight quads at a time before any of their stores, so the loads overlap.
  auto val = [&](int h, int j, int e) {  // row rm + 32 h + e, column j of this thread's 8 H
    // the half that holds row e's product: row 0 leads in acc[0], row 1 in acc[1]
    const int s = (e ^ j) & 1, half = s ? 1 - (e & 1) : e & 1;
    return __uint_as_float((unsigned)(acc[s][2 * h + (e >> 1)][j >> 1] >> (32 * half)));
  };
  const bool vec = tri == 0 && ((uintptr_t)C % 16 == 0) && (ldc % 4 == 0) && m0 + BM <= M && n0 + BN <= N;
  if (vec) {
#pragma unroll
    for (int jh = 0; jh < 8 * H; jh += 4) {  // rounds of 4 H float4 loads, then their stores
      float4 cv[4][H];
#pragma unroll
      for (int jj = 0; jj < 4; jj++)
#pragma unroll
        for (int h = 0; h < H; h++) {
          const int c = n0 + cn + 4 * jh + jj, r = m0 + rm + 32 * h;
          cv[jj][h] = beta != 0.f ? *reinterpret_cast<const float4 *>(C + r + (long)c * ldc)
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
      for (int jj = 0; jj < 4; jj++)
#pragma unroll
        for (int h = 0; h < H; h++) {
          const int j = jh + jj, c = n0 + cn + 4 * jh + jj, r = m0 + rm + 32 * h;
          float4 o;
          o.x = alpha * val(h, j, 0);
          o.y = alpha * val(h, j, 1);
          o.z = alpha * val(h, j, 2);
          o.w = alpha * val(h, j, 3);
          if (beta != 0.f) {
            o.x = fmaf(beta, cv[jj][h].x, o.x);
            o.y = fmaf(beta, cv[jj][h].y, o.y);
            o.z = fmaf(beta, cv[jj][h].z, o.z);
            o.w = fmaf(beta, cv[jj][h].w, o.w);
          }
          *reinterpret_cast<float4 *>(C + r + (long)c * ldc) = o;
        }
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 8 * H; j++) {
    const int c = n0 + cn + 16 * (j >> 2) + (j & 3);
    float cv[4 * H];
#pragma unroll
    for (int i = 0; i < 4 * H; i++) {
      const int r = m0 + rm + (i < 4 ? i : 32 + i - 4);
      const bool ok = r < M && c < N && !(tri == 1 && r < c) && !(tri == 2 && r > c);
      cv[i] = (ok && beta != 0.f) ? C[r + (long)c * ldc] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4 * H; i++) {
      const int r = m0 + rm + (i < 4 ? i : 32 + i - 4);
      if (r >= M || c >= N) continue;
      if (tri == 1 && r < c) continue;
      if (tri == 2 && r > c) continue;
      float v = alpha * val(i >> 2, j, i & 3);
      if (beta != 0.f) v = fmaf(beta, cv[i], v);
      C[r + (long)c * ldc] = v;
    }
  }
}

// C = beta C + alpha (sum of the S partial products in W, ld M), in C's triangle
__global__ void splitk_sum_kernel(int M, int N, int S, const float *__restrict__ W, float alpha, float beta,
                                  float *__restrict__ C, long ldc, int tri) {
  const long total = (long)M * N;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
    const int r = (int)(idx % M), c = (int)(idx / M);
    if (tri == 1 && r < c) continue;
    if (tri == 2 && r > c) continue;
    float v = 0.f;
    for (int s = 0; s < S; s++) v += W[idx + (long)s * total];
    float *p = C + r + (long)c * ldc;
    *p = beta == 0.f ? alpha * v : fmaf(beta, *p, alpha * v);
  }
}

__global__ void sscale_kernel(int M, int N, float beta, float *C, long ldc, int tri) {
  long idx = blockIdx.x * (long)blockDim.x + threadIdx.x;
  long total = (long)M * N;
  for (; idx < total; idx += (long)gridDim.x * blockDim.x) {
    int r = (int)(idx % M), c = (int)(idx / M);
    if (tri == 1 && r < c) continue;
    if (tri == 2 && r > c) continue;
    float *p = C + r + (long)c * ldc;
    *p = (beta == 0.f) ? 0.f : beta * *p;
  }
}

}  // namespace

void sgemm_dev(int ta, int tb, int M, int N, int K, float alpha, const float *A, long lda,
               const float *B, long ldb, float beta, float *C, long ldc, cudaStream_t st,
               int tri) {
  if (M <= 0 || N <= 0) return;
  if (K <= 0 || alpha == 0.f) {
    if (beta == 1.f) return;
    long total = (long)M * N;
    int blocks = (int)std::min<long>((total + 255) / 256, 148L * 16);
    sscale_kernel<<<blocks, 256, 0, st>>>(M, N, beta, C, ldc, tri);
    ATLB_CUDA_CHECK(cudaGetLastError());
    return;
  }
  const int tiles = cdiv(M, BT) * cdiv(N, BT);
  const bool tA = ta != kNoTrans, tB = tb != kNoTrans;
  // few output tiles and a long K: split K so that about two CTAs per SM run
  int S = 1, kc = K;
  float *W = nullptr;
  if (tiles < num_sms() / 2 && K >= 1024 && !no_alloc_active()) {
    S = std::min(cdiv(K, 256), std::max(1, 2 * num_sms() / tiles));
    kc = cdiv(cdiv(K, S), BK) * BK;
    S = cdiv(K, kc);
    if (S > 1) W = (float *)scratch(kSlotGemmSplit, sizeof(float) * (size_t)S * M * N);
    else kc = K;
  }
  // 16-byte copies need the outer index contiguous and 16-byte aligned columns
  const bool va = !tA && (uintptr_t)A % 16 == 0 && lda % 4 == 0, vb = tB && (uintptr_t)B % 16 == 0 && ldb % 4 == 0;
  auto with = [&](auto tile) {
    constexpr int T = decltype(tile)::value;
    auto go = [&](auto kern, bool &configured) {
      if (!configured) {
        ATLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem<T>));
        ATLB_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
        configured = true;
      }
      kern<<<dim3(cdiv(M, T) * cdiv(N, T), S), THREADS, kSmem<T>, st>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc,
                                                                         tri, kc, W);
    };
    static bool set[9] = {};
    if (!tA && !tB) {
      if (va) go(sgemm_simt_kernel<T, false, false, true, false>, set[0]);
      else go(sgemm_simt_kernel<T, false, false, false, false>, set[1]);
    } else if (!tA && tB) {
      if (va && vb) go(sgemm_simt_kernel<T, false, true, true, true>, set[2]);
      else if (va) go(sgemm_simt_kernel<T, false, true, true, false>, set[3]);
      else if (vb) go(sgemm_simt_kernel<T, false, true, false, true>, set[4]);
      else go(sgemm_simt_kernel<T, false, true, false, false>, set[5]);
    } else if (tA && !tB) {
      go(sgemm_simt_kernel<T, true, false, false, false>, set[6]);
    } else {
      if (vb) go(sgemm_simt_kernel<T, true, true, false, true>, set[7]);
      else go(sgemm_simt_kernel<T, true, true, false, false>, set[8]);
    }
  };
  const bool few = 4 * tiles <= 3 * num_sms() || (K <= 128 && tiles < num_sms());
  if (S == 1 && few) with(std::integral_constant<int, 64>{});
  else with(std::integral_constant<int, BT>{});
  ATLB_CUDA_CHECK(cudaGetLastError());
  if (S > 1) {
    const long total = (long)M * N;
    splitk_sum_kernel<<<(int)std::min<long>((total + 255) / 256, 148L * 8), 256, 0, st>>>(M, N, S, W, alpha, beta, C,
                                                                                      ldc, tri);
    ATLB_CUDA_CHECK(cudaGetLastError());
  }
}

}  // namespace atlb
