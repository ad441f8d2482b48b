// crgpu_smem.h - dynamic shared-memory limits of the kernels (host code only).
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <utility>

namespace crgpu {

// Raises a kernel's dynamic shared-memory limit on the current device to at least `bytes` and never
// lowers it.  The attribute belongs to the process and the device, not to a stream or a solver: setting
// it to each launch's own size would let a smaller solve on another host thread shrink it under a
// larger one's launch, which then fails (or, for a kernel whose output is read without its own error
// check, leaves stale data).
inline cudaError_t raise_smem_limit(const void* kernel, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> set;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    size_t& cur = set[{device, kernel}];
    if (bytes <= cur) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

}  // namespace crgpu
