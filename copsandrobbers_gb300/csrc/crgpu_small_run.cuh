// crgpu_small_run.cuh - the kernel of crgpu_small.cu for one number of cops (CR_SMALL_K), a translation
// unit each so that they compile side by side.
#include <cuda_runtime.h>

#define CR_SMALL_NS2(k) small##k
#define CR_SMALL_NS(k) CR_SMALL_NS2(k)
#define CR_BODY_NS CR_SMALL_NS(CR_SMALL_K)
#define CR_LDG(p) (*(p))
#define CR_RESTRICT
#define CR_BODY_INLINE __noinline__
#include "crgpu_v1_body.cuh"
#include "crgpu_small.cuh"
#include "crgpu_team.cuh"

namespace crgpu {
namespace CR_BODY_NS {

// A pass's end: its count (or the error bits) to the ring, column 0's prep for the next one, and
// whether there is one.  By one thread, between two barriers.
__device__ __noinline__ void end_pass(const V1Dev& d, const LoopCtl& c, int i) {
    const unsigned err = *d.err;
    const unsigned long long found = *d.pass_new;
    *(volatile unsigned long long*)(c.hist + (i & (c.ring - 1))) = err ? kHistError | err : found;
    *d.done = err || !found ? 1u : 0u;
    prep_reset(d, 0, 1);
}

template <int K, int RWP, bool P1>
__device__ void run_passes(const V1Dev& d, const LoopCtl& c, const Team& tm, int first, int passes) {
    constexpr int G = RWP <= 4 ? 4 : RWP;
    constexpr int NWP = RWP * 2;
    const unsigned wk = tm.rank, nwk = tm.size;
    const bool lead = tm.thread() == 0;
    // as k_loop_enter: column 1's list after a fused first pass, column 0's prep, the first count
    if (d.meta[1].compact) team_list_compact(tm, d, 1);
    prep_clear(d, 0, wk, nwk);
    tm.sync();
    if (lead) {
        d.meta[1].compact = 0;
        if (first) {
            end_pass(d, c, 0);
        } else {
            *d.done = 0u;
            prep_reset(d, 0, 1);
        }
    }
    tm.sync();
    for (int i = first; i < passes; ++i) {
        if (*(volatile unsigned*)d.done) break;   // (the same word for every thread, between barriers)
        for (int col = 0; col < d.cols; ++col) {
            const int nx = (col + 1) % d.cols;
            if (col % 2 == 0) {
                const ColMeta mi = d.meta[nx];
                const bool some = mi.hi >= mi.lo;
                if (mi.seed) {
                    cop_seed_body<K, G>(d, col, nx, wk, nwk);
                    tm.sync();
                } else if (frontier_sparse(d, mi)) {
                    cop_push_body<K>(d, col, nx, wk, nwk);
                    tm.sync();
                    if (some) {
                        cop_apply_body<G>(d, col, nx, wk, nwk);
                        tm.sync();
                    }
                } else if (some) {
                    if constexpr (K >= 2) {
                        head_rows_body<K, RWP>(d, nx, wk, nwk);
                        tm.sync();
                        sep_pull_body<K, RWP>(d, col, nx, wk, nwk);
                    } else {
                        cop_pull_body<K, NWP, G>(d, col, nx, wk, nwk);
                    }
                    tm.sync();
                }
                prep_clear_flags(d, nx, wk, nwk);
                tm.sync();
                if (lead) prep_reset(d, nx, (nx + 1) % d.cols);
                tm.sync();
            } else {
                prep_clear_cand(d, wk, nwk);
                if (col < d.cols - 1) direct_body<G>(d, col, nx, wk, nwk);
                else last_column_body<P1, G>(d, col, wk, nwk);
                tm.sync();
                if (lead) {
                    if (col < d.cols - 1) prep_reset(d, nx, (nx + 1) % d.cols);
                    else end_pass(d, c, i);
                }
                tm.sync();
            }
        }
    }
}

template <int K>
__global__ void __launch_bounds__(kSmallThreads, 1) k_small_run(V1Dev d, LoopCtl c, int first, int passes, int p1) {
    Team tm;
    tm.of_cluster();
    switch (d.g.rwp) {
        case 1:
            if (p1) run_passes<K, 1, true>(d, c, tm, first, passes);
            else run_passes<K, 1, false>(d, c, tm, first, passes);
            break;
        case 2:
            if (p1) run_passes<K, 2, true>(d, c, tm, first, passes);
            else run_passes<K, 2, false>(d, c, tm, first, passes);
            break;
        case 4:
            if (p1) run_passes<K, 4, true>(d, c, tm, first, passes);
            else run_passes<K, 4, false>(d, c, tm, first, passes);
            break;
        default:
            if (p1) run_passes<K, 8, true>(d, c, tm, first, passes);
            else run_passes<K, 8, false>(d, c, tm, first, passes);
            break;
    }
}

template <int K>
cudaError_t launch_small_k(const V1Dev& d, const LoopCtl& c, int first, int passes, bool p1, int team, size_t sm, cudaStream_t st) {
    if (sm > 40 * 1024) {
        const cudaError_t e = raise_smem_limit((const void*)k_small_run<K>, sm);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)team);
    cfg.blockDim = dim3(kSmallThreads);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)team;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_small_run<K>, d, c, first, passes, p1 ? 1 : 0);
}

}  // namespace CR_BODY_NS

template <>
cudaError_t launch_small<CR_SMALL_K>(const V1Dev& d, const LoopCtl& c, int first, int passes, bool p1, int team, size_t sm,
                                     cudaStream_t st) {
    return CR_BODY_NS::launch_small_k<CR_SMALL_K>(d, c, first, passes, p1, team, sm, st);
}

}  // namespace crgpu
