// crgpu_small.cuh - what crgpu_small.cu and its per-k translation units share.
#pragma once
#include "crgpu_internal.cuh"

namespace crgpu {

constexpr int kSmallThreads = 512;

// Launches k_small_run<K> with `team` blocks as one cluster and `sm` bytes of dynamic shared memory.
template <int K>
cudaError_t launch_small(const V1Dev& d, const LoopCtl& c, int first, int passes, bool p1, int team, size_t sm, cudaStream_t st);
template <> cudaError_t launch_small<1>(const V1Dev&, const LoopCtl&, int, int, bool, int, size_t, cudaStream_t);
template <> cudaError_t launch_small<2>(const V1Dev&, const LoopCtl&, int, int, bool, int, size_t, cudaStream_t);
template <> cudaError_t launch_small<3>(const V1Dev&, const LoopCtl&, int, int, bool, int, size_t, cudaStream_t);
template <> cudaError_t launch_small<4>(const V1Dev&, const LoopCtl&, int, int, bool, int, size_t, cudaStream_t);

}  // namespace crgpu
