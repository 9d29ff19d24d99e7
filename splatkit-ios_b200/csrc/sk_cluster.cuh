// Thread-block clusters: the hardware barrier of a cluster's blocks and stores into their shared memory.
//
// A block's shared memory may be written by another block only once it is known to have started, which
// being scheduled together does not say: every kernel arrives at the cluster barrier as its first
// instruction and waits for it before its first storeRemote. The wait is over by then as a rule (the
// kernel's loads and first sums lie in between).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace sk {

__device__ __forceinline__ void clusterArrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void clusterWait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t clusterRank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Stores to the word at `p` of this block's shared memory, in block `rank` of the cluster.
__device__ __forceinline__ void storeRemote(uint32_t* p, uint32_t rank, uint32_t v) {
  const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  asm volatile(
      "{\n\t.reg .u32 a;\n\t"
      "mapa.shared::cluster.u32 a, %0, %1;\n\t"
      "st.shared::cluster.u32 [a], %2;\n\t}" ::"r"(at),
      "r"(rank), "r"(v)
      : "memory");
}

}  // namespace sk
