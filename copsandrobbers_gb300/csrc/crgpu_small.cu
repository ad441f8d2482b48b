// crgpu_small.cu - the passes of a small v1 solve in one launch.
//
// A pass of a small solve is a few microseconds of work behind three launches per visibility step,
// each of which costs as much again, and a wait for its count.  Here one thread-block cluster (or a
// single block) runs the passes of a solve one after the other, the same bodies as the stand-alone
// kernels (crgpu_v1_body.cuh) as workers 0 .. size-1 with cluster barriers between them, until a
// pass finds nothing, an error bit is set or the asked number has run.  The counts go to the same
// ring as those of k_and_end.  Nothing waits for anything outside the cluster.
#include <cuda_runtime.h>

#include <algorithm>

#define CR_BODY_NS small0
#define CR_LDG(p) (*(p))
#define CR_RESTRICT
#define CR_BODY_INLINE __noinline__
#include "crgpu_v1_body.cuh"
#include "crgpu_small.cuh"

namespace crgpu {

using namespace small0;   // (the bodies' shared-memory sizes)

// Dynamic shared memory of k_small_run: the largest need of its bodies.
static size_t small_smem(int k, int n, int rw, int rwp, int S) {
    const int warps = kSmallThreads / 32, G = rwp <= 4 ? 4 : rwp, CPW = 32 / G;
    const size_t cop = (size_t)warps * CPW * 2 * S * rwp + rank_table_words(k, n);
    const size_t rows = (size_t)warps * CPW * and_group_words(S, rwp);
    const size_t heads = (size_t)head_smem_words(kSmallThreads, k, n, rwp);
    const size_t tile = (size_t)warps * and_tile_quads(rw) * 4;
    return std::max(std::max(cop, rows), std::max(heads, tile)) * 4;
}

// Blocks of the team that runs a solve's passes, 0 = the solve is not small.  Work of a dense pass in
// row words: per configuration the rows of its successor heads and about eight more.  Whole runs by
// launches, by one block and by a cluster of eight (us): 4-regular n = 24, k = 2, p = 3 (3.8 K words)
// 100, 66, 86; Delaunay n = 199, k = 1 (14 K) 236, 151, 185; n = 48, k = 2 (29 K) 338, 407, 310; n = 20,
// k = 3, p = 2 (44 K) 366, 493, 336; n = 26, k = 3 (91 K) 196, 541, 224.
int small_team(const V1Dev& d, double avg_deg) {
    if (d.g.n > 256 || d.S != 2 || (d.k >= 2 && !d.h1)) return 0;
    double heads = 1;
    for (int i = 1; i < d.k; ++i) heads *= avg_deg;
    const double words = (double)d.C * d.g.rwp * (8 + heads);
    if (words > 4.8e4 || small_smem(d.k, d.g.n, d.g.rw, d.g.rwp, d.S) > 200 * 1024) return 0;
    return words > 1.6e4 ? 8 : 1;
}

// Passes first .. passes - 1 of a solve by a team of small_team() blocks (first = 1: a fused first
// pass has just run and is recorded as pass 0).
cudaError_t launch_small_run(const V1Dev& d, const LoopCtl& c, int first, int passes, bool p1, int team, cudaStream_t st) {
    const size_t sm = small_smem(d.k, d.g.n, d.g.rw, d.g.rwp, d.S);
    switch (d.k) {
        case 1: return launch_small<1>(d, c, first, passes, p1, team, sm, st);
        case 2: return launch_small<2>(d, c, first, passes, p1, team, sm, st);
        case 3: return launch_small<3>(d, c, first, passes, p1, team, sm, st);
        default: return launch_small<4>(d, c, first, passes, p1, team, sm, st);
    }
}

}  // namespace crgpu
