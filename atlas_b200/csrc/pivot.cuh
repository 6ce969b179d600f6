// Pivot search by integer keys: the panel kernels of the LU factorizations
// (lu.cu, batched.cu).
#pragma once
#include <cuda_runtime.h>
#include <type_traits>

namespace atlb {

template <typename T>
using PivKey = typename std::conditional<sizeof(T) == 8, unsigned long long, unsigned>::type;

// Candidates are compared through one integer key: |value|'s bit pattern + 1
// (non-negative IEEE values order like their bit patterns), 0 for a NaN or
// for "no candidate"; ties go to the lowest row position.  A warp's arg-max
// is then three redux instructions instead of a shuffle tree.
template <typename T>
__device__ __forceinline__ unsigned long long pivot_key(T v) {
  const T t = fabs(v);
  if (!(t >= T(0))) return 0ull;
  if (sizeof(T) == 8) return (unsigned long long)__double_as_longlong((double)t) + 1ull;
  return (unsigned long long)__float_as_uint((float)t) + 1ull;
}
__device__ __forceinline__ void warp_argmax_key(unsigned &key, unsigned &pos) {  // FP32 keys fit 32 bits
  const unsigned m = __reduce_max_sync(0xffffffffu, key);
  pos = __reduce_min_sync(0xffffffffu, key == m ? pos : 0xffffffffu);
  key = m;
}
__device__ __forceinline__ void warp_argmax_key(unsigned long long &key, unsigned &pos) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? lo : 0u);
  const bool eq = hi == mhi && lo == mlo;
  pos = __reduce_min_sync(0xffffffffu, eq ? pos : 0xffffffffu);
  key = ((unsigned long long)mhi << 32) | mlo;
}

// Lane of the warp's largest key (lowest pos among equal keys).  Usually
// the high 32 bits of the largest key occur in one lane only: one redux and
// one ballot then settle it.
template <typename K>
__device__ __forceinline__ int warp_argmax_lane(K key, unsigned pos) {
  const unsigned hi = sizeof(K) == 8 ? (unsigned)((unsigned long long)key >> 32) : (unsigned)key;
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned m = __ballot_sync(0xffffffffu, hi == mhi);
  if ((m & (m - 1)) == 0) return __ffs(m) - 1;
  K k = key;
  unsigned p = pos;
  warp_argmax_key(k, p);
  return __ffs(__ballot_sync(0xffffffffu, key == k && pos == p)) - 1;
}

}  // namespace atlb
