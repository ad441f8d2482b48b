// crgpu_team.cuh - the blocks that solve one graph together: one, or a thread-block cluster.
#pragma once
#include <cuda_runtime.h>

namespace crgpu {

struct Team {
    unsigned rank, size;
    __device__ __forceinline__ void of_cluster() {
        asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
        asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    }
    // Every thread of the team, with the memory effects of __syncthreads over all of it (the cluster
    // barrier's arrive releases and its wait acquires at cluster scope).
    __device__ __forceinline__ void sync() const {
        __syncthreads();
        if (size > 1) {
            asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        }
    }
    __device__ __forceinline__ unsigned thread() const { return rank * blockDim.x + threadIdx.x; }
    __device__ __forceinline__ unsigned threads() const { return size * blockDim.x; }
};

}  // namespace crgpu
