// Words passed between the CTAs of a thread-block cluster (sm_103a).
#pragma once
#include <cuda_runtime.h>

constexpr int kClusterPolls = 1 << 22;   // bound of every wait on another CTA: about 0.1 s in shared memory, 3 s in global memory

__device__ __forceinline__ void st_cluster(void* p, unsigned long long v) {   // p: generic address of cluster shared memory
  asm volatile("st.relaxed.cluster.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(int* p, int v) {
  asm volatile("st.relaxed.cluster.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// polls of words in this CTA's own shared memory
__device__ __forceinline__ int ld_poll(const int* p) {
  int v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
  return v;
}
__device__ __forceinline__ void fence_cluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
// Release of this CTA's own shared memory and acquire of the cluster's (30 to
// 70 cycles, where a full fence.acq_rel.cluster took 950).
__device__ __forceinline__ void fence_release_shared() {
  asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_acquire_shared() {
  asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
}
