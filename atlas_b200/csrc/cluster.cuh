// Messages between the CTAs of a cluster without a cluster barrier: one-way
// stores that complete a transaction on the receiver's mbarrier (the panel
// kernels of lu.cu and qr.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

namespace atlb {

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t a, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
// one-way 16-byte store into another CTA's shared memory that completes a
// transaction on that CTA's mbarrier (no fence, no round trip)
__device__ __forceinline__ void st_async16(uint32_t addr, uint4 v, uint32_t mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(mbar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t a, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
               " selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(a), "r"(parity) : "memory");
  return ok != 0;
}
// the same, 8 bytes
__device__ __forceinline__ void st_async8(uint32_t addr, double v, uint32_t mbar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
               ::"r"(addr), "l"(__double_as_longlong(v)), "r"(mbar) : "memory");
}

}  // namespace atlb
