// crgpu_team.cuh - the blocks that solve one graph together: one, or a thread-block cluster.
#pragma once
#include <cuda_runtime.h>

#include "crgpu_internal.cuh"

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

// Column col's row list from its flag plane, by the whole team (after the fused first pass).
__device__ __noinline__ inline void team_list_compact(const Team& tm, const V1Dev& d, int col) {
    const uint8_t* f = d.fflag + (size_t)col * d.C;
    uint32_t* out = d.list + (size_t)col * d.C;
    const int lane = threadIdx.x & 31;
    for (uint32_t base = tm.thread() & ~31u; base < d.C; base += tm.threads()) {
        const uint32_t i = base + lane;
        const bool set = i < d.C && f[i];
        const unsigned b = __ballot_sync(0xFFFFFFFFu, set);
        if (!b) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(&d.meta[col].len, __popc(b));
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
        if (set) out[at + __popc(b & ((1u << lane) - 1u))] = i;
    }
}

}  // namespace crgpu
