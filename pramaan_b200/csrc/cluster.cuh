// cluster.cuh — what the cluster kernels share: the plain CSR they read and
// the cluster's registers and barrier.
#pragma once

#include "common.cuh"

namespace pb {

struct FlatCsr {
    const int* row_ptr;
    const int* col;
    const float* val;
};

__device__ __forceinline__ unsigned cluster_rank_in() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_blocks() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_index_x() {
    unsigned r;
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace pb
