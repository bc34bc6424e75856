// cluster_ptx.cuh -- the hardware barrier of a thread-block cluster.
#pragma once
#include <stdint.h>

namespace pgd_cl {

// Waits for every thread of the cluster; writes before it (shared or global) are
// visible to the cluster's reads after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

}  // namespace pgd_cl
