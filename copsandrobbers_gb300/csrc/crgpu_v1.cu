// crgpu_v1.cu - level-synchronous frontier kernels for the v1 rules
// (solvers/k_cops_visibility.cpp: 2p DP columns per visibility cycle).
//
// The reference sweeps all C*N*2p states every pass, column 0 to 2p-1, in place
// (k_cops_visibility.cpp:142-296).  Within one column every state reads only the next
// column, so the order inside a column is irrelevant and one pass is exactly: each column c
// in turn recomputed from column c+1 as it stood before this pass (c+1 is recomputed later
// in the pass), except the last column, which reads column 0 as just recomputed.  These
// kernels run that same schedule, but a column's producer only looks at the states whose
// inputs changed: the marks column c+1's last producer run made (its frontier).
//
//   cop turn (even c)          (C, r, c) = 1 + min over C' in T(C) of marked (C', r, c+1)
//                              k_cops_visibility.cpp:160-197
//   deferred robber (odd c)    (C, r, c) = 1 + (C, r, c+1)           k_cops_visibility.cpp:209-228
//   last column (2p-1)         (C, r, 2p-1) = 1 + max over v p hops from r of (C, v, 0), all
//                              marked                              k_cops_visibility.cpp:235-288
// with values >= 127 left unmarked (lines 189, 220, 280).
//
// Why frontiers suffice: a state left unmarked after its producer ran had no marked input
// then, or every marked input already gave a value >= 127.  Values in a column never
// decrease from one pass to the next, so any input that can now mark it is a new one, and
// the minimum over new inputs equals the minimum over all inputs whenever it is < 127.
// The frontier of a column is split into value slots (one bit plane per value) so that the
// cop-turn minimum is a sequence of bitwise ORs: the lowest slot with a bit gives the value.
//
// The cop turn runs in one of these forms, chosen on the device from the frontier's row count:
//   seed          the capture seeds of column 1 before pass 1, in closed form: the OR of the
//                 seed rows over T(C) is the union of the cops' neighbourhoods;
//   pull (dense)  every configuration ORs the frontier rows of its successors: for k = 2, 3, 4
//                 in separable form through head rows (head_rows + sep_pull), else one by one
//                 (k_cop_pull);
//   push (sparse) every row of the frontier's list is ORed into the candidate rows of its
//                 predecessors with atomics, then only those rows are marked (push + apply).
// k_cop_a and k_cop_b carry the seed, push, apply and separable bodies (each body returns at
// once unless its form applies), so a cop turn is two launches with head rows and three without.
#include "crgpu_internal.cuh"

#include <algorithm>

#define CR_BODY_NS grid
#define CR_LDG(p) __ldg(p)
#define CR_RESTRICT __restrict__
#define CR_BODY_INLINE __forceinline__
#include "crgpu_v1_body.cuh"

namespace crgpu {

using namespace grid;

__device__ void list_compact_body(const V1Dev& d, int col);

// The kernels of a pass are short and each waits for the one before it, so they are launched with
// programmatic stream serialisation: a kernel's blocks are placed while its predecessor drains, and
// wait here before they touch memory.  False = nothing to do (behind the fixed point).
__device__ __forceinline__ bool pass_kernel_begin(const V1Dev& d) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    return !d.done || *d.done == 0u;
}

__global__ void k_prep(V1Dev d, int col, int nx) { prep_body(d, col, nx, blockIdx.x, gridDim.x); }
// initializeCaptures; with `whole` also the columns without captures (marked rows and flags cleared, so
// that only the table's bytes are left to a clear) and the state of a fresh solve: capture seeds in
// columns 0 and 1 (every row, the implicit list), pass 1's column-0 producer appending to column 0's.
__global__ void k_init(V1Dev d, int K, bool whole) {
    if (whole) {
        if (blockIdx.x == 0) {
            const int rows = d.C < 0x7FFFFFFFu ? (int)d.C : 0x7FFFFFFF;
            for (int c = threadIdx.x; c < d.cols; c += blockDim.x)
                d.meta[c] = c == 0   ? ColMeta{0, 0, 0, 1, rows, 0, -1, 0}
                            : c == 1 ? ColMeta{0, 0, 0, 0, rows, 1, -1, 0}
                                     : ColMeta{0, kEmptyLo, -1, 0, 0, 0, 0, 0};
            if (threadIdx.x < kSyncWords) d.sync[threadIdx.x] = 0u;
            if (threadIdx.x == 0) *d.err = 0u;
        }
        const size_t flags = (size_t)(d.cols - 2) * d.C, words = flags * d.g.rwp;
        const size_t step = (size_t)gridDim.x * blockDim.x, first = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
        for (size_t i = first; i < flags; i += step) d.fflag[2 * (size_t)d.C + i] = 0;
        uint32_t* m = d.marked + 2 * (size_t)d.C * d.g.rwp;
        if (d.g.rwp & 3) {
            for (size_t i = first; i < words; i += step) m[i] = 0u;
        } else {
            for (size_t i = first; i < words / 4; i += step) reinterpret_cast<uint4*>(m)[i] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    init_body(d, K, blockIdx.x, gridDim.x);
}
// The first pass in three forms (launch_init_pass1): the run form of rows of one 256-robber block
// split into whole lane pieces with byte masks (at most 85 registers, 3 blocks of 256 per SM, which
// measured faster than 64 registers at 4 blocks and than 2 blocks), the tiles, and the general sweep
// (64 registers).
template <int K, int W, bool SINGLE>
__global__ void __launch_bounds__(256, SINGLE ? 3 : 4) k_init_pass1(V1Dev d) {
    if (SINGLE) {
        if (d.g.n == 256) init_pass1_single<K, W, true>(d, blockIdx.x, gridDim.x);
        else init_pass1_single<K, W, false>(d, blockIdx.x, gridDim.x);
    } else {
        init_pass1_body<K, W>(d, blockIdx.x, gridDim.x);
    }
}
template <int K>
__global__ void __launch_bounds__(256, 3) k_init_tiles(V1Dev d) {
    if ((d.g.n & 15) == 0) init_pass1_tiles<K, true>(d, blockIdx.x, gridDim.x);
    else init_pass1_tiles<K, false>(d, blockIdx.x, gridDim.x);
}

template <int K, int NWP, int G>
__global__ void __launch_bounds__(256) k_cop_pull(V1Dev d, int col, int nx) {
    if (!pass_kernel_begin(d)) return;
    cop_pull_body<K, NWP, G>(d, col, nx, blockIdx.x, gridDim.x);
}
// The other cop-turn forms share two launches, each body returning at once unless its form
// applies (the form is chosen on the device from the input frontier):
//   k_cop_a  the capture-seed form, the push scatter, or the separable turn's head rows;
//   k_cop_b  the separable turn's configurations or the push form's marking.
// The tuple-gathering pull (k = 1, or no head rows) keeps its own launch: it wants up to 127
// registers; k_cop_a at most 64 (80 with 32-word rows), k_cop_b up to 85, which keep the rows of four
// successor heads in flight (Delaunay n = 199: 5.5 ms of cop turns, 5.7 at 64 registers with spills).
template <int K, int NWP, int G>
__global__ void __launch_bounds__(256, NWP >= 32 ? 3 : 4) k_cop_a(V1Dev d, int col, int nx) {
    if (!pass_kernel_begin(d)) return;
    cop_seed_body<K, G>(d, col, nx, blockIdx.x, gridDim.x);
    cop_push_body<K>(d, col, nx, blockIdx.x, gridDim.x);
    if constexpr (K >= 2) head_rows_body<K, NWP / 2>(d, nx, blockIdx.x, gridDim.x);
}
template <int K, int NWP, int G>
__global__ void __launch_bounds__(256, 3) k_cop_b(V1Dev d, int col, int nx) {
    if (!pass_kernel_begin(d)) return;
    if constexpr (K >= 2) sep_pull_body<K, NWP / 2>(d, col, nx, blockIdx.x, gridDim.x);
    cop_apply_body<G>(d, col, nx, blockIdx.x, gridDim.x);
}
// k_cop_b followed by the prep of the column it consumed (nx): the flags a dense turn left there
// (no body of this launch reads them), and in the last block the column's state reset.  The
// candidate rows wait for that column's producer.
template <int K, int NWP, int G>
__global__ void __launch_bounds__(256, 3) k_cop_b_end(V1Dev d, int col, int nx) {
    if (!pass_kernel_begin(d)) return;
    if constexpr (K >= 2) sep_pull_body<K, NWP / 2>(d, col, nx, blockIdx.x, gridDim.x);
    cop_apply_body<G>(d, col, nx, blockIdx.x, gridDim.x);
    prep_clear_flags(d, nx, blockIdx.x, gridDim.x);
    __syncthreads();
    if (threadIdx.x == 0 && grid_last_block(d, gridDim.x)) prep_reset(d, nx, (nx + 1) % d.cols);
}
// The deferred robber turn; with `end` also the rest of its own prep (the candidate rows) and, in
// the last block, the prep of column nx, whose frontier it consumed (every listed flag cleared).
template <int G>
__global__ void __launch_bounds__(256) k_direct(V1Dev d, int col, int nx, bool end) {
    if (!pass_kernel_begin(d)) return;
    if (end) prep_clear_cand(d, blockIdx.x, gridDim.x);
    direct_body<G>(d, col, nx, blockIdx.x, gridDim.x);
    if (!end) return;
    __syncthreads();
    if (threadIdx.x == 0 && grid_last_block(d, gridDim.x)) prep_reset(d, nx, (nx + 1) % d.cols);
}
// The last column, with the end of the pass in its last block: the pass's count goes to the host's
// ring, and column 0's prep for the next pass runs (this column cleared every flag of column 0's
// list, so that prep is a reset of the column's state).
// At most 64 registers: the grid runs 4 blocks of 256 per SM (more registers cost occupancy
// that the latency-bound row forms need more).
template <bool P1, int G>
__global__ void __launch_bounds__(256, 4) k_and_end(V1Dev d, int col, LoopCtl c) {
    if (!pass_kernel_begin(d)) return;
    if (c.hist) prep_clear_cand(d, blockIdx.x, gridDim.x);   // this column's prep, the rest
    last_column_body<P1, G>(d, col, blockIdx.x, gridDim.x);
    if (!c.hist) return;
    __syncthreads();
    if (threadIdx.x == 0 && grid_last_block(d, gridDim.x)) {
        const int i = *c.idx;
        const unsigned err = *d.err;
        volatile unsigned long long* word = c.hist + (i & (c.ring - 1));
        if (err) {
            *word = kHistError | err;
        } else {
            const unsigned long long found = *d.pass_new;
            *word = found;
            *c.idx = i + 1;
            if (!found) *d.done = 1u;
        }
        prep_reset(d, 0, 1);
    }
}

// Before the first of the passes of a call: column 1's row list after a fused first pass (every block
// reads the marker before the last block clears it), column 0's prep (again, harmlessly, when an
// earlier call's last pass ran it), and in the last block the history, which a first pass run
// just before opens with its count.
__global__ void __launch_bounds__(256) k_loop_enter(V1Dev d, LoopCtl c, int first) {
    if (d.meta[1].compact) list_compact_body(d, 1);
    prep_clear(d, 0, blockIdx.x, gridDim.x);
    __syncthreads();
    if (threadIdx.x == 0 && grid_last_block(d, gridDim.x)) {
        d.meta[1].compact = 0;
        const unsigned err = *d.err;
        if (first) *(volatile unsigned long long*)c.hist = err ? kHistError | err : *d.pass_new;
        *c.idx = first;
        *d.done = first && !*d.pass_new ? 1u : 0u;
        prep_reset(d, 0, 1);
    }
}

__global__ void k_verdict(const uint8_t* __restrict__ table, const uint32_t* __restrict__ m0,
                          uint32_t C, int n, int rw, int rwp, int cols, unsigned long long* best) {
    verdict_body(table, m0, C, n, rw, rwp, cols, best, blockIdx.x, gridDim.x);
}

// ---------------------------------------------------------------- host-side launchers ---



// Lanes per configuration: a power of two covering the robber row (at least 4).
static int group_lanes(int rwp) {
    int g = 4;
    while (g < rwp) g <<= 1;
    return g;
}

size_t cop_smem_bytes(int S, int rwp) {
    return (size_t)8 * (32 / group_lanes(rwp)) * 2 * S * rwp * sizeof(uint32_t);
}
size_t and_smem_bytes(int S, int rwp, int n) {
    (void)n;
    return (size_t)8 * (32 / group_lanes(rwp)) * and_group_words(S, rwp) * sizeof(uint32_t);
}
// Eight warps of the last column's tile form.
static size_t and_tile_smem_bytes(int rw) { return (size_t)8 * and_tile_quads(rw) * 16; }

static int pull_words(int S, int rwp) {
    int w = S * rwp, p = 2;
    while (p < w) p <<= 1;
    return p;
}

bool pull_supported(int S, int rwp) { return pull_words(S, rwp) <= 32 && group_lanes(rwp) <= 32; }

template <typename... P, typename... A>
static void launch_pass_kernel(void (*kernel)(P...), int grid, size_t sm, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute serial = {};
    serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    serial.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &serial;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

template <int K, int NWP, int G>
static void launch_cop_ng(const V1Dev& d, int col, int nx, int grid, cudaStream_t st, bool end) {
    const size_t sm = cop_smem_bytes(d.S, d.g.rwp);
    const size_t smr = sm + (size_t)rank_table_words(K, d.g.n) * 4;
    const size_t sma = d.h1 ? std::max(smr, (size_t)head_smem_words(256, K, d.g.n, d.g.rwp) * 4) : smr;
    if (sma > 40 * 1024) raise_smem_limit((const void*)k_cop_a<K, NWP, G>, sma);   // (plus the static part)
    launch_pass_kernel(k_cop_a<K, NWP, G>, grid, sma, st, d, col, nx);
    if (!d.h1) launch_pass_kernel(k_cop_pull<K, NWP, G>, grid, smr, st, d, col, nx);
    // (three blocks of k_cop_b per SM are resident, four of the other kernels)
    const int grid_b = grid - grid / 4;
    launch_pass_kernel(end ? k_cop_b_end<K, NWP, G> : k_cop_b<K, NWP, G>, grid_b, sm, st, d, col, nx);
}

// Accumulator words and lanes per configuration, as the pull and the separable turn use them.
template <int K>
static void launch_cop_k(const V1Dev& d, int col, int nx, int grid, cudaStream_t st, bool end) {
    const int G = group_lanes(d.g.rwp);
    switch (pull_words(d.S, d.g.rwp)) {
        case 2: launch_cop_ng<K, 2, 4>(d, col, nx, grid, st, end); break;
        case 4: launch_cop_ng<K, 4, 4>(d, col, nx, grid, st, end); break;
        case 8: launch_cop_ng<K, 8, 4>(d, col, nx, grid, st, end); break;
        case 16:
            if (G == 4) launch_cop_ng<K, 16, 4>(d, col, nx, grid, st, end);
            else launch_cop_ng<K, 16, 8>(d, col, nx, grid, st, end);
            break;
        default:
            if (G == 4) launch_cop_ng<K, 32, 4>(d, col, nx, grid, st, end);
            else if (G == 8) launch_cop_ng<K, 32, 8>(d, col, nx, grid, st, end);
            else launch_cop_ng<K, 32, 16>(d, col, nx, grid, st, end);
            break;
    }
}

template <int G>
static void launch_direct_g(const V1Dev& d, int col, int nx, int grid, cudaStream_t st, bool end) {
    launch_pass_kernel(k_direct<G>, grid, cop_smem_bytes(d.S, d.g.rwp), st, d, col, nx, end);
}

// Cop turn into column col (or, direct = 1, a deferred robber turn): every form that may apply
// is enqueued; each reads the input frontier's row count on the device and only the matching
// form does work.
void launch_cop(const V1Dev& d, int col, int nx, int direct, int grid, cudaStream_t st, bool end) {
    if (direct) {
        switch (group_lanes(d.g.rwp)) {
            case 4: launch_direct_g<4>(d, col, nx, grid, st, end); break;
            case 8: launch_direct_g<8>(d, col, nx, grid, st, end); break;
            case 16: launch_direct_g<16>(d, col, nx, grid, st, end); break;
            default: launch_direct_g<32>(d, col, nx, grid, st, end); break;
        }
        return;
    }
    switch (d.k) {
        case 1: launch_cop_k<1>(d, col, nx, grid, st, end); break;
        case 2: launch_cop_k<2>(d, col, nx, grid, st, end); break;
        case 3: launch_cop_k<3>(d, col, nx, grid, st, end); break;
        default: launch_cop_k<4>(d, col, nx, grid, st, end); break;
    }
}

int cop_launches(int direct) { return direct ? 1 : 3; }
int cop_launches_k(int direct, bool sep) { return direct ? 1 : (sep ? 2 : 3); }

// Shared-memory words the last-column body stages the graph in: transposed hop rows, row
// pointers and neighbour lists.
size_t and_stage_words(int n, int rwp, int nnz) {
    return (size_t)n * rwp + n + 1 + (size_t)(nnz + 1) / 2;
}

template <bool P1, int G>
static void launch_and_g(const V1Dev& d, int col, int grid, size_t sm, cudaStream_t st, const LoopCtl& loop) {
    if (sm > 40 * 1024) raise_smem_limit((const void*)k_and_end<P1, G>, sm);   // (plus the static part)
    launch_pass_kernel(k_and_end<P1, G>, grid, sm, st, d, col, loop);
}

template <bool P1>
static void launch_and_p(const V1Dev& d0, int col, int grid, cudaStream_t st, const LoopCtl& loop) {
    V1Dev d = d0;
    size_t sm = and_smem_bytes(d.S, d.g.rwp, d.g.n);
    d.and_stage_words = 0;
    if (d.g.nnz >= 0) {
        const size_t words = and_stage_words(d.g.n, d.g.rwp, d.g.nnz);
        if (sm + words * 4 <= 48 * 1024) {   // within the default dynamic shared-memory limit
            d.and_stage_words = (uint32_t)words;
            sm += words * 4;
        }
    }
    if (d.g.ell) sm = std::max(sm, and_tile_smem_bytes(d.g.rw));
    switch (group_lanes(d.g.rwp)) {
        case 4: launch_and_g<P1, 4>(d, col, grid, sm, st, loop); break;
        case 8: launch_and_g<P1, 8>(d, col, grid, sm, st, loop); break;
        case 16: launch_and_g<P1, 16>(d, col, grid, sm, st, loop); break;
        default: launch_and_g<P1, 32>(d, col, grid, sm, st, loop); break;
    }
}

void launch_and(const V1Dev& d, int col, bool p1, int grid, cudaStream_t st, const LoopCtl& loop) {
    if (p1) launch_and_p<true>(d, col, grid, st, loop);
    else launch_and_p<false>(d, col, grid, st, loop);
}

void launch_loop_enter(const V1Dev& d, const LoopCtl& c, int first, int grid, cudaStream_t st) {
    k_loop_enter<<<grid, 256, 0, st>>>(d, c, first);
}

void launch_prep(const V1Dev& d, int col, int nx, int grid, cudaStream_t st) {
    k_prep<<<grid, 256, 0, st>>>(d, col, nx);
}

void launch_init(const V1Dev& d, bool whole, int grid, cudaStream_t st) { k_init<<<grid, 256, 0, st>>>(d, d.k, whole); }

template <int W, bool SINGLE>
static void launch_init_pass1_w(const V1Dev& d, int grid, size_t sm, cudaStream_t st) {
    switch (d.k) {
        case 1: k_init_pass1<1, W, SINGLE><<<grid, 256, sm, st>>>(d); break;
        case 2: k_init_pass1<2, W, SINGLE><<<grid, 256, sm, st>>>(d); break;
        case 3: k_init_pass1<3, W, SINGLE><<<grid, 256, sm, st>>>(d); break;
        default: k_init_pass1<4, W, SINGLE><<<grid, 256, sm, st>>>(d); break;
    }
}
// Requires d.g.cover (cover_w 1, 2 or 4) and two columns.  Three forms, one wave of resident blocks:
//   run      rows of one 256-robber block split into whole lane pieces, at most 8 neighbours, at
//            least 3: column 1 then hardly marks anything in this pass, and the run form's test of
//            that is the cheapest (4-regular n = 256, k = 3: 300 us, tiles 490 us);
//   tiles    every other graph of 16 vertices and more whose cops can all move: where robbers with
//            one or two neighbours are caught in most configurations the run form leaves its fast
//            loop for each of them (G(n, p) n = 128, k = 3: 159 us, tiles 80 us), and the general
//            sweep writes rows that are not 16-byte aligned byte by byte (Delaunay n = 199 1760 us,
//            tiles 340; n = 389 25.0 and 3.8 ms; G(n, p) n = 61, k = 4 519 and 105 us);
//   general  the rest.
template <int K>
static void launch_init_tiles(const V1Dev& d, int num_sms, cudaStream_t st) {
    const size_t sm = (size_t)pass1_tile_words(8, d.g.n, d.g.rw) * 4;
    if (sm > 40 * 1024) raise_smem_limit((const void*)k_init_tiles<K>, sm);
    const int per_sm = std::max(1, std::min(3, (int)(220 * 1024 / (sm + 1024))));
    const uint64_t cap = ((uint64_t)d.C + 31) / 32;
    k_init_tiles<K><<<(int)std::max<uint64_t>(1, std::min<uint64_t>(cap, (uint64_t)num_sms * per_sm)), 256, sm, st>>>(d);
}

void launch_init_pass1(const V1Dev& d, int num_sms, cudaStream_t st) {
    const bool run = d.g.n <= 256 && (d.g.n & 7) == 0 && d.g.cover_w == 1 && (d.g.mindeg >= 3 || !d.g.cin);
    if (!run && d.g.cin && d.g.ell) {
        switch (d.k) {
            case 1: launch_init_tiles<1>(d, num_sms, st); break;
            case 2: launch_init_tiles<2>(d, num_sms, st); break;
            case 3: launch_init_tiles<3>(d, num_sms, st); break;
            default: launch_init_tiles<4>(d, num_sms, st); break;
        }
        return;
    }
    const uint64_t cap = ((uint64_t)d.C + 7) / 8;
    const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>(cap, (uint64_t)num_sms * (run ? 3 : 4)));
    if (run) launch_init_pass1_w<1, true>(d, grid, (size_t)init_pass1_smem_words(d.g.n, d.g.rwp) * 4, st);
    else if (d.g.cover_w == 1) launch_init_pass1_w<1, false>(d, grid, 0, st);
    else if (d.g.cover_w == 2) launch_init_pass1_w<2, false>(d, grid, 0, st);
    else launch_init_pass1_w<4, false>(d, grid, 0, st);
}

// Builds column col's row list from its flag plane (after the first pass): each block takes
// segments of 16 flags per thread, counts the set ones, reserves its segment's room in the list
// with one atomic and writes the ids (the list order is irrelevant to its consumers).
__device__ void list_compact_body(const V1Dev& d, int col) {
    __shared__ unsigned s_warp[8];
    __shared__ unsigned s_at;
    constexpr int kPer = 16;
    const uint8_t* f = d.fflag + (size_t)col * d.C;
    uint32_t* out = d.list + (size_t)col * d.C;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t seg = (size_t)blockDim.x * kPer;
    for (size_t base = (size_t)blockIdx.x * seg; base < d.C; base += (size_t)gridDim.x * seg) {
        unsigned bits = 0;   // bit j: flag base + j * blockDim.x + threadIdx.x is set
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const size_t i = base + (size_t)j * blockDim.x + threadIdx.x;
            if (i < d.C && f[i]) bits |= 1u << j;
        }
        const unsigned mine = __popc(bits);
        unsigned incl = mine;   // inclusive scan over the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned tot = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
                const unsigned c = s_warp[w];
                s_warp[w] = tot;
                tot += c;
            }
            s_at = tot ? (unsigned)atomicAdd(&d.meta[col].len, (int)tot) : 0u;
        }
        __syncthreads();
        unsigned at = s_at + s_warp[warp] + incl - mine;
        while (bits) {
            const int j = __ffs(bits) - 1;
            bits &= bits - 1;
            out[at++] = (uint32_t)(base + (size_t)j * blockDim.x + threadIdx.x);
        }
        __syncthreads();
    }
}
void launch_verdict(const V1Dev& d, int cols, unsigned long long* best, int grid, cudaStream_t st) {
    k_verdict<<<grid, 256, 0, st>>>(d.table, d.marked, d.C, d.g.n, d.g.rw, d.g.rwp, cols, best);
}

void launch_verdict_raw(const uint8_t* table, const uint32_t* m0, uint32_t C, int n, int rw,
                        int rwp, int cols, unsigned long long* best, int grid, cudaStream_t st) {
    k_verdict<<<grid, 256, 0, st>>>(table, m0, C, n, rw, rwp, cols, best);
}

int max_cop_blocks_per_sm(int k, int rwp, int S) {
    // grid-stride kernels: 4 blocks of 256 per SM keep every SM busy whatever the
    // register count of the instance (blocks beyond residency simply queue)
    (void)k; (void)rwp; (void)S;
    return 4;
}

}  // namespace crgpu
