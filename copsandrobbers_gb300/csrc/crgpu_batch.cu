// crgpu_batch.cu - many small solves in one persistent launch.
//
// The batched workload is the cop number of many small graphs: for each graph solve k = 1, 2,
// 3 ... in order (v1 rules) and stop at the first WIN.  Solved one launch sequence at a time,
// a small graph costs a few microseconds of work per pass but tens of microseconds of launch
// and synchronisation, so the GPU idles.  Here one persistent kernel owns the whole batch:
// each thread block takes the next graph from a device-side queue (graphs ordered by cost,
// largest first), solves its k = 1, 2, ... sequence itself in a private slot of device memory,
// and writes a result per (graph, k): verdict, pass counts digest and a table digest.  The
// block runs the same frontier bodies as the stand-alone kernels (crgpu_v1_body.cuh) with
// (worker 0 of 1), separated by __syncthreads, so its tables are the same bytes.
//
// A graph of 128 vertices keeps one block busy for a quarter of a second, so a batch that does not
// hold many times more graphs than the GPU has blocks would wait for the last large ones.  The
// batch is therefore split: its largest graphs are solved first by teams of 2, 4 or 8 blocks (a
// thread-block cluster, the bodies running as workers 0 .. size-1 with cluster barriers between
// them), then every block goes on alone through the smaller ones.  How many graphs the teams take
// and how large the teams are comes from a model of the batch's run time (plan_teams).  No block
// ever waits for one outside its cluster; the only state shared beyond it are the queue counters.
//
// The block size and blocks per SM are chosen by a small autotuner that times candidate
// launch shapes on a calibration slice of the batch (cached per device and batch shape).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <tuple>
#include <vector>

#define CR_BODY_NS cta
#define CR_LDG(p) (*(p))
#define CR_RESTRICT
#define CR_BODY_INLINE __noinline__
#include "../../include/crgpu.h"
#include "crgpu_batch_plan.h"
#include "crgpu_ctx.h"
#include "crgpu_v1_body.cuh"
#include "crgpu_team.cuh"

namespace crgpu {

size_t and_stage_words(int n, int rwp, int nnz);

using namespace cta;

constexpr int kBatchMaxN = 128;
constexpr int kBatchMaxK = 3;

struct BatchDev {
    int count, kmax, p;
    const int32_t* order;
    const int32_t* n;
    const int32_t* maxdeg;
    const uint64_t* rp_off;   // per graph: offset of its n+1 row pointers in rp_all / rrp_all
    const uint64_t* col_off;  // per graph: offset of its neighbour lists in col_all / rcol_all
    const uint32_t* rp_all;
    const uint16_t* col_all;
    const uint32_t* rrp_all;
    const uint16_t* rcol_all;
    unsigned char* slots;
    size_t team_bytes;             // a team's slot, and a block's share of it once it goes alone
    size_t solo_bytes;
    int team_count;                // order[0 .. team_count) are the teams'
    int* next;                     // [0] the teams' queue, [1] the single blocks'
    int* mail;                     // per team: the graph it took
    int32_t* cop;
    cr_batch_result* res;
    unsigned long long* cta_time;  // per block: globaltimer at start and after its last graph
    uint32_t smem_words;           // dynamic shared memory of the launch
};

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// 64-bit mixer (the splitmix64 finaliser of Steele, Lea and Flood) used by the table digest.
__host__ __device__ inline uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__host__ __device__ inline uint64_t binom_dev(int64_t n, int64_t k) {
    if (k < 0 || n < 0 || k > n) return 0;
    if (k > n - k) k = n - k;
    uint64_t r = 1;
    for (int64_t i = 1; i <= k; ++i) r = r * (uint64_t)(n - i + 1) / (uint64_t)i;
    return r;
}

// Byte offsets of one (n, k, p) solve inside a slot.
struct JobLayout {
    size_t binom, configs, nbr, iso, hop, rhop, ell, ell_off, cover, table, marked, front, h1, list, clist, fflag, cand,
        cbits, sync, meta, counters, err, total;
};

__host__ __device__ inline JobLayout job_layout(int n, int k, int p, int S) {
    const uint64_t C = binom_dev((int64_t)n + k - 1, k);
    const int rwp = round_words((n + 31) / 32), cols = 2 * p;
    JobLayout L;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off += (bytes + 255) & ~size_t(255);
        return at;
    };
    L.binom = take((size_t)k * (n + 1) * 4);
    L.configs = take(C * k * 2);
    L.nbr = take((size_t)n * rwp * 4);
    L.iso = take((size_t)rwp * 4);
    L.hop = take((size_t)n * rwp * 4);
    L.rhop = take((size_t)n * rwp * 4);
    // neighbour lists of the last column's tile form: 32 side by side, each up to n long
    L.ell = take((size_t)((n + 31) / 32) * 32 * n * 2);
    L.ell_off = take((size_t)((n + 31) / 32 + 1) * 4);
    // uncovered-slot masks of the fused first pass (p = 1), up to 4 bytes per mask
    L.cover = take(p == 1 ? 2 * (size_t)n * ((n + 7) & ~7) * 4 : 0);
    L.table = take(C * (size_t)n * cols);
    L.marked = take((size_t)cols * C * rwp * 4);
    L.front = take((size_t)cols * C * S * rwp * 4);
    // k = 2, 3: head rows of the separable dense cop turn (written before they are read each
    // pass, so they sit outside the regions the block zeroes)
    L.h1 = take(k >= 2 ? (size_t)binom_dev((int64_t)n + k - 2, k - 1) * n * S * rwp * 4 : 0);
    // frontier row lists and the push-mode candidate list (written before they are read)
    L.list = take((size_t)cols * C * 4);
    L.clist = take(C * 4);
    L.fflag = take((size_t)cols * C);
    L.cand = take(C * S * rwp * 4);
    L.cbits = take(cand_bits_bytes(C));
    L.sync = take(kSyncWords * sizeof(unsigned));
    L.meta = take(sizeof(ColMeta) * cols);
    L.counters = take(4 * sizeof(unsigned long long));
    L.err = take(sizeof(unsigned));
    L.total = off;
    return L;
}

// Table digest: sum over 8-byte little-endian words w_j (zero-padded tail) of
// mix64(w_j ^ (j * 0x9E3779B97F4A7C15)), modulo 2^64.
__device__ inline uint64_t digest_word(const uint8_t* t, size_t bytes, size_t j) {
    uint64_t w = 0;
    const size_t at = j * 8;
    if (at + 8 <= bytes && ((uintptr_t)t & 7u) == 0) {
        w = *reinterpret_cast<const uint64_t*>(t + at);   // little-endian: byte b at bits 8b
    } else if (at + 8 <= bytes) {
        for (int b = 0; b < 8; ++b) w |= (uint64_t)t[at + b] << (8 * b);
    } else {
        for (size_t b = 0; at + b < bytes; ++b) w |= (uint64_t)t[at + b] << (8 * b);
    }
    return mix64(w ^ (j * 0x9E3779B97F4A7C15ull));
}

__device__ void team_fill(const Team& tm, unsigned char* p, unsigned char v, size_t bytes) {
    // p is 256-byte aligned (slot layout)
    const uint32_t v4 = 0x01010101u * v;
    const uint4 q = make_uint4(v4, v4, v4, v4);
    uint4* p16 = reinterpret_cast<uint4*>(p);
    const size_t n16 = bytes / 16;
    for (size_t i = tm.thread(); i < n16; i += tm.threads()) p16[i] = q;
    for (size_t i = n16 * 16 + tm.thread(); i < bytes; i += tm.threads()) p[i] = v;
}

// The uncovered-slot masks of the fused first pass, as the stand-alone solver builds them on the
// host (cover[c][r] bit j: r's j-th neighbour v is neither c nor a neighbour of c; cover[n+c][r]:
// v is not c; a cop's own entry all ones, the rows of a cop without a move zero), W = 1, 2 or 4
// bytes per mask by the largest degree.  Sets d.g.cover, cover_w and npad.
__device__ void build_cover(const Team& tm, V1Dev& d, uint8_t* cov, int maxdeg) {
    const int n = d.g.n, rwp = d.g.rwp, npad = (n + 7) & ~7;
    const int W = maxdeg <= 8 ? 1 : (maxdeg <= 16 ? 2 : 4);
    const uint32_t ones = W == 4 ? 0xFFFFFFFFu : ((1u << (8 * W)) - 1u);
    const size_t plane = (size_t)n * npad * W;
    for (int t = tm.thread(); t < n * npad; t += tm.threads()) {
        const int c = t / npad, r = t - c * npad;
        uint32_t m0 = 0, m1 = 0;
        if (r < n) {
            const uint32_t e0 = d.g.row_ptr[r], deg = d.g.row_ptr[r + 1] - e0;
            for (uint32_t j = 0; j < deg; ++j) {
                const int v = d.g.col[e0 + j];
                if (v == c) continue;
                m1 |= 1u << j;
                if (!((d.g.nbr[(size_t)c * rwp + (v >> 5)] >> (v & 31)) & 1u)) m0 |= 1u << j;
            }
            if (r == c) m0 = ones;
        }
        if ((d.g.isolated[c >> 5] >> (c & 31)) & 1u) m0 = 0;
        for (int q = 0; q < W; ++q) {
            cov[(size_t)t * W + q] = (uint8_t)(m0 >> (8 * q));
            cov[plane + (size_t)t * W + q] = (uint8_t)(m1 >> (8 * q));
        }
    }
    d.g.cover = cov;
    d.g.cover_w = W;
    d.g.npad = npad;
    tm.sync();
}

// The padded neighbour lists of the last column's tile form (d.g.ell): row word w's 32 lists
// take as many rows as the longest of them.  The team's first block builds them, a warp for every
// word (n <= 128).
__device__ void build_ell(const Team& tm, V1Dev& d, uint16_t* ell, uint32_t* off) {
    d.g.ell = ell;
    d.g.ell_off = off;
    if (tm.rank != 0) {
        tm.sync();
        return;
    }
    const int n = d.g.n, rw = d.g.rw, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = warp * 32 + lane;
    uint32_t e0 = 0, deg = 0;
    if (r < n) {
        e0 = d.g.row_ptr[r];
        deg = d.g.row_ptr[r + 1] - e0;
    }
    const uint32_t longest = __reduce_max_sync(0xFFFFFFFFu, deg);
    if (warp < rw && lane == 0) off[warp + 1] = longest;
    __syncthreads();
    if (threadIdx.x == 0) {
        off[0] = 0;
        for (int w = 0; w < rw; ++w) off[w + 1] += off[w];
    }
    __syncthreads();
    if (warp < rw) {
        uint16_t* at = ell + (size_t)off[warp] * 32 + lane;
        for (uint32_t e = 0; e < longest; ++e) at[e * 32] = e < deg ? d.g.col[e0 + e] : (uint16_t)(rw * 32);
    }
    tm.sync();
}

// One (graph, k) solve by a team.  Returns 1 on WIN.
template <int K, int RWP, bool P1>
__device__ int solve_job(const BatchDev& b, const Team& tm, unsigned char* slot, int gi, int jr) {
    constexpr int G = RWP <= 4 ? 4 : RWP;
    constexpr int NWP = RWP * 2 <= 2 ? 2 : RWP * 2;  // S = 2 slots
    const int n = b.n[gi], p = b.p, cols = 2 * p, S = 2;
    const int rw = (n + 31) / 32, rwp = round_words(rw);
    const uint64_t C = binom_dev((int64_t)n + K - 1, K);
    const JobLayout L = job_layout(n, K, p, S);
    V1Dev d;
    d.g.n = n;
    d.g.maxdeg = b.maxdeg[gi];
    d.g.rw = rw;
    d.g.rwp = rwp;
    d.g.row_ptr = b.rp_all + b.rp_off[gi];
    d.g.col = b.col_all + b.col_off[gi];
    d.g.rrow_ptr = b.rrp_all + b.rp_off[gi];
    d.g.rcol = b.rcol_all + b.col_off[gi];
    d.g.nbr = reinterpret_cast<const uint32_t*>(slot + L.nbr);
    d.g.isolated = reinterpret_cast<const uint32_t*>(slot + L.iso);
    d.g.rhop = reinterpret_cast<const uint32_t*>(slot + L.rhop);
    d.k = K;
    d.cols = cols;
    d.S = S;
    d.C = (uint32_t)C;
    d.binom = reinterpret_cast<const uint32_t*>(slot + L.binom);
    d.configs = reinterpret_cast<const uint16_t*>(slot + L.configs);
    d.hop = reinterpret_cast<const uint32_t*>(slot + L.hop);
    d.table = slot + L.table;
    d.marked = reinterpret_cast<uint32_t*>(slot + L.marked);
    d.front = reinterpret_cast<uint32_t*>(slot + L.front);
    d.fflag = slot + L.fflag;
    d.cand = reinterpret_cast<uint32_t*>(slot + L.cand);
    d.h1 = K >= 2 ? reinterpret_cast<uint32_t*>(slot + L.h1) : nullptr;
    if (d.h1) d.push_ratio = kPushRatioSeparable;
    d.cbits = reinterpret_cast<uint32_t*>(slot + L.cbits);
    d.list = reinterpret_cast<uint32_t*>(slot + L.list);
    d.clist = reinterpret_cast<uint32_t*>(slot + L.clist);
    d.sync = reinterpret_cast<unsigned*>(slot + L.sync);
    d.meta = reinterpret_cast<ColMeta*>(slot + L.meta);
    d.pass_new = reinterpret_cast<unsigned long long*>(slot + L.counters);
    d.err = reinterpret_cast<unsigned*>(slot + L.err);
    {
        // room past the last-column body's lane groups for staging the graph
        constexpr int CPW = 32 / G;
        const uint32_t groups = (blockDim.x >> 5) * CPW * and_group_words(S, rwp);
        d.and_stage_words = b.smem_words > groups ? b.smem_words - groups : 0u;
    }
    uint32_t* binom = reinterpret_cast<uint32_t*>(slot + L.binom);
    uint32_t* nbr = reinterpret_cast<uint32_t*>(slot + L.nbr);
    uint32_t* iso = reinterpret_cast<uint32_t*>(slot + L.iso);
    uint32_t* hop = reinterpret_cast<uint32_t*>(slot + L.hop);
    uint16_t* configs = reinterpret_cast<uint16_t*>(slot + L.configs);

    // initializeCaptures and pass 1 fused (as the stand-alone p = 1 solve does) when the
    // uncovered-slot masks fit: the first pass then writes every table byte and both marked
    // planes itself
    const int maxdeg = b.maxdeg[gi];
    const bool fused = P1 && maxdeg <= 32;
    // ---- buildAuxGraph: zeroed planes, rank table, neighbour masks, configurations
    team_fill(tm, slot + L.nbr, 0, L.ell - L.nbr);
    if (!fused) {
        team_fill(tm, slot + L.marked, 0, L.front - L.marked);
        team_fill(tm, d.table, kUnmarked, C * (size_t)n * cols);
    }
    team_fill(tm, slot + L.fflag, 0, L.total - L.fflag);
    const int np1 = n + 1;
    for (int t = tm.thread(); t < K * np1; t += tm.threads()) {
        const int i = t / np1, x = t - i * np1;
        binom[t] = (uint32_t)binom_dev((int64_t)n - x + K - 1 - i, K - i);
    }
    tm.sync();
    for (int u = tm.thread(); u < n; u += tm.threads()) {
        const uint32_t e0 = d.g.row_ptr[u], e1 = d.g.row_ptr[u + 1];
        if (e0 == e1) atomicOr(&iso[u >> 5], 1u << (u & 31));
        for (uint32_t e = e0; e < e1; ++e) {
            const int v = d.g.col[e];
            nbr[(size_t)u * rwp + (v >> 5)] |= 1u << (v & 31);
        }
        // transposed 1-hop masks: the in-neighbours of u
        uint32_t* rh = reinterpret_cast<uint32_t*>(slot + L.rhop) + (size_t)u * rwp;
        for (uint32_t e = d.g.rrow_ptr[u]; e < d.g.rrow_ptr[u + 1]; ++e) {
            const int r = d.g.rcol[e];
            rh[r >> 5] |= 1u << (r & 31);
        }
    }
    for (uint32_t cid = tm.thread(); cid < C; cid += tm.threads()) {
        uint32_t rem = cid;
        int prev = 0;
        for (int i = 0; i < K; ++i) {
            const uint32_t top = binom[i * np1 + prev];
            int lo = prev, hi = n - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (binom[i * np1 + mid] >= top - rem) lo = mid; else hi = mid - 1;
            }
            rem -= top - binom[i * np1 + lo];
            configs[(size_t)cid * K + i] = (uint16_t)lo;
            prev = lo;
        }
    }
    tm.sync();
    if (P1) build_ell(tm, d, reinterpret_cast<uint16_t*>(slot + L.ell), reinterpret_cast<uint32_t*>(slot + L.ell_off));
    if (!P1) {
        for (int r = tm.thread(); r < n; r += tm.threads()) {
            uint32_t cur[kBatchMaxN / 32], nxt[kBatchMaxN / 32];
            for (int w = 0; w < rwp; ++w) cur[w] = 0u;
            cur[r >> 5] = 1u << (r & 31);
            for (int s = 0; s < p; ++s) {
                for (int w = 0; w < rwp; ++w) nxt[w] = 0u;
                for (int w = 0; w < rwp; ++w) {
                    uint32_t bb = cur[w];
                    while (bb) {
                        const int v = w * 32 + __ffs(bb) - 1;
                        bb &= bb - 1;
                        for (int q = 0; q < rwp; ++q) nxt[q] |= nbr[(size_t)v * rwp + q];
                    }
                }
                for (int w = 0; w < rwp; ++w) cur[w] = nxt[w];
            }
            for (int w = 0; w < rwp; ++w) hop[(size_t)r * rwp + w] = cur[w];
        }
    }
    uint64_t caps = 0, phash = 0;
    int passes = 0;
    bool more = true;
    if (fused) {
        build_cover(tm, d, slot + L.cover, maxdeg);
        if (tm.thread() == 0) {
            for (int c = 0; c < cols; ++c) d.meta[c] = ColMeta{0, kEmptyLo, -1, 0, 0, 0, 0, 0};
            d.meta[0] = ColMeta{0, 0, 0, 0, (int)C, 0, -1, 1};   // consumed: flags left clear
            d.meta[1] = ColMeta{1, kEmptyLo, -1, 0, 0, 0, 0, 0};
        }
        tm.sync();
        if (d.g.cover_w == 1) init_pass1_body<K, 1>(d, tm.rank, tm.size);
        else if (d.g.cover_w == 2) init_pass1_body<K, 2>(d, tm.rank, tm.size);
        else init_pass1_body<K, 4>(d, tm.rank, tm.size);
        tm.sync();
        team_list_compact(tm, d, 1);
        tm.sync();
        // every configuration's distinct cops: n times the multisets holding a given vertex
        caps = (uint64_t)n * (binom_dev((int64_t)n + K - 1, K) - binom_dev((int64_t)n + K - 2, K));
        const uint64_t found = *d.pass_new;
        const unsigned bits = *d.err;
        tm.sync();
        passes = 1;
        phash = mix64(found ^ (1ull * 0xD1B54A32D192ED03ull));
        more = found != 0 && !bits;
    } else {
        // ---- initializeCaptures
        if (tm.thread() == 0) {
            for (int c = 0; c < cols; ++c) d.meta[c] = ColMeta{0, kEmptyLo, -1, 0, 0, 0, 0, 0};
            d.meta[0] = ColMeta{0, 0, 0, 1, (int)C, 0, -1, 0};
            d.meta[1] = ColMeta{0, 0, 0, 0, (int)C, 1, -1, 0};
        }
        tm.sync();
        init_body(d, K, tm.rank, tm.size);
        tm.sync();
        caps = *d.pass_new;
        tm.sync();
    }
    // ---- mainLoop
    while (more) {
        for (int col = 0; col < cols; ++col) {
            const int nx = (col + 1) % cols;
            prep_body(d, col, nx, tm.rank, tm.size);
            tm.sync();
            if (col % 2 == 0) {
                cop_seed_body<K, G>(d, col, nx, tm.rank, tm.size);
                tm.sync();
                if constexpr (K == 1) {
                    cop_pull_body<K, NWP, G>(d, col, nx, tm.rank, tm.size);
                    tm.sync();
                }
                if constexpr (K >= 2) {
                    head_rows_body<K, RWP>(d, nx, tm.rank, tm.size);
                    tm.sync();
                    sep_pull_body<K, RWP>(d, col, nx, tm.rank, tm.size);
                    tm.sync();
                }
                cop_push_body<K>(d, col, nx, tm.rank, tm.size);
                tm.sync();
                cop_apply_body<G>(d, col, nx, tm.rank, tm.size);
            } else if (col < cols - 1) {
                direct_body<G>(d, col, nx, tm.rank, tm.size);
            } else {
                last_column_body<P1, G>(d, col, tm.rank, tm.size);
            }
            tm.sync();
        }
        const uint64_t found = *d.pass_new;
        const unsigned bits = *d.err;
        tm.sync();
        ++passes;
        phash += mix64(found ^ ((uint64_t)passes * 0xD1B54A32D192ED03ull));
        if (bits || found == 0 || passes >= 4096) break;
    }
    // ---- findFinalResult
    unsigned long long* best = d.pass_new + 1;   // then the digest, and whether the cops win
    if (tm.thread() == 0) *best = ~0ull;
    tm.sync();
    verdict_body(d.table, d.marked, d.C, n, rw, rwp, cols, best, tm.rank, tm.size);
    // ---- table digest
    const size_t bytes = C * (size_t)n * cols;
    uint64_t part = 0;
    for (size_t j = tm.thread(); j < (bytes + 7) / 8; j += tm.threads()) part += digest_word(d.table, bytes, j);
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(d.pass_new + 2, (unsigned long long)part);
    tm.sync();
    if (tm.thread() == 0) {
        const unsigned long long key = *best;
        cr_batch_result& r = b.res[jr];
        r.solved = 1;
        r.status = *d.err ? CR_ERR_INTERNAL : (passes >= 4096 ? CR_ERR_BUDGET : CR_OK);
        const int won = (key != ~0ull && (int)(key >> 32) < kMaxRound) ? 1 : 0;
        r.win = won;
        r.capture_plies = won ? (int32_t)(key >> 32) : kMaxRound;
        r.best_config = won ? (int64_t)(key & 0xFFFFFFFFull) : -1;
        r.passes = passes;
        r.base_captures = caps;
        r.states = C * (uint64_t)n * cols;
        r.digest = d.pass_new[2];
        r.pass_hash = phash;
        d.pass_new[3] = (unsigned long long)won;
    }
    tm.sync();
    const int win = (int)*(volatile unsigned long long*)(d.pass_new + 3);
    tm.sync();
    return win;
}

template <int K, bool P1>
__device__ int solve_job_k(const BatchDev& b, const Team& tm, unsigned char* slot, int gi, int jr) {
    const int rwp = round_words((b.n[gi] + 31) / 32);
    if (rwp <= 1) return solve_job<K, 1, P1>(b, tm, slot, gi, jr);
    if (rwp <= 2) return solve_job<K, 2, P1>(b, tm, slot, gi, jr);
    return solve_job<K, 4, P1>(b, tm, slot, gi, jr);
}

// Two builds: up to 512 threads per block with up to 128 registers (no spills in the bodies),
// and 1024 threads with 64 (a few spills, twice the threads on each graph).
template <bool P1>
__device__ void solve_graph(const BatchDev& b, const Team& tm, unsigned char* slot, int gi) {
    int cop = 0;
    for (int k = 1; k <= b.kmax; ++k) {
        const int jr = gi * b.kmax + (k - 1);
        int win;
        if (k == 1) win = solve_job_k<1, P1>(b, tm, slot, gi, jr);
        else if (k == 2) win = solve_job_k<2, P1>(b, tm, slot, gi, jr);
        else win = solve_job_k<3, P1>(b, tm, slot, gi, jr);
        if (win) { cop = k; break; }
    }
    if (tm.thread() == 0) b.cop[gi] = cop;
    if (threadIdx.x == 0) b.cta_time[2 * blockIdx.x + 1] = global_ns();
}

template <bool P1, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_batch(BatchDev b) {
    __shared__ int s_job;
    Team tm;
    tm.of_cluster();
    const unsigned team = blockIdx.x / tm.size;
    unsigned char* slot = b.slots + (size_t)team * b.team_bytes;
    if (threadIdx.x == 0) b.cta_time[2 * blockIdx.x] = b.cta_time[2 * blockIdx.x + 1] = global_ns();
    // the teams' graphs
    for (;;) {
        if (tm.thread() == 0) b.mail[team] = atomicAdd(&b.next[0], 1);
        tm.sync();
        const int jj = *(volatile int*)(b.mail + team);
        tm.sync();
        if (jj >= b.team_count) break;
        solve_graph<P1>(b, tm, slot, b.order[jj]);
    }
    // the others, a block each, in its share of the team's slot
    slot += tm.rank * b.solo_bytes;
    const Team solo{0u, 1u};
    for (;;) {
        if (threadIdx.x == 0) s_job = atomicAdd(&b.next[1], 1);
        __syncthreads();
        const int jj = b.team_count + s_job;
        __syncthreads();
        if (jj >= b.count) break;
        solve_graph<P1>(b, solo, slot, b.order[jj]);
    }
}

// Grid-wide digest of a stand-alone solver's table (same function as the batch's).
__global__ void k_digest(const uint8_t* table, size_t bytes, unsigned long long* out) {
    uint64_t part = 0;
    for (size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x; j < (bytes + 7) / 8;
         j += (size_t)gridDim.x * blockDim.x)
        part += digest_word(table, bytes, j);
    for (int off = 16; off > 0; off >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, off);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, (unsigned long long)part);
}

void launch_digest(const uint8_t* table, size_t bytes, unsigned long long* out, int grid, cudaStream_t st) {
    k_digest<<<grid, 256, 0, st>>>(table, bytes, out);
}

}  // namespace crgpu

using namespace crgpu;

namespace {

// Dynamic shared memory of the batch kernel: the largest need over every vertex count up to
// max_n (lane groups, and so the per-group footprint, change with the row width).
size_t batch_smem(int threads, int max_n) {
    size_t best = 0;
    for (int n = 1; n <= max_n; ++n) {
        const int rwp = round_words((n + 31) / 32);
        const int G = rwp <= 4 ? 4 : rwp, CPW = 32 / G, warps = threads / 32, S = 2;
        const size_t cop = (size_t)warps * CPW * 2 * S * rwp;
        const size_t andb = (size_t)warps * CPW * and_group_words(S, rwp);
        const size_t push = (size_t)warps * S * rwp;
        const size_t pull = cop + rank_table_words(kBatchMaxK, n);
        const size_t head = (size_t)head_smem_words(threads, kBatchMaxK, n, rwp);
        const size_t tile = (size_t)warps * and_tile_quads((n + 31) / 32) * 4;
        best = std::max(best, std::max(std::max(std::max(pull, head), tile), std::max(andb, push)) * 4);
    }
    return best;
}

struct Shape {
    int threads, per_sm;
};

std::mutex g_tune_mu;
std::map<std::tuple<int, int, int, int>, Shape> g_tuned;

int fail(cr_context* ctx, int code, const char* msg) {
    if (ctx) ctx->err = msg;
    return code;
}

}  // namespace

#define CR_BCUDA(call)                                                                     \
    do {                                                                                   \
        cudaError_t e_ = (call);                                                           \
        if (e_ != cudaSuccess) {                                                           \
            ctx->err = std::string(#call) + ": " + cudaGetErrorString(e_);                 \
            return e_ == cudaErrorMemoryAllocation ? CR_ERR_NOMEM : CR_ERR_CUDA;           \
        }                                                                                  \
    } while (0)

namespace {

// Device copies of one batch's inputs.
struct BatchInputs {
    std::vector<int32_t> n, maxdeg, order;
    std::vector<uint64_t> rp_off, col_off;
    std::vector<uint32_t> rp, rrp;
    std::vector<uint16_t> col, rcol;
    int max_n = 0;
    size_t max_stage_words = 0;   // the largest graph staging of the last-column body
};

using BatchKernel = void (*)(BatchDev);
BatchKernel batch_kernel(Shape shape) { return shape.threads > 512 ? k_batch<true, 1024> : k_batch<true, 512>; }

size_t launch_smem(const BatchInputs& in, Shape shape) {
    return batch_smem(shape.threads, in.max_n) + in.max_stage_words * 4;
}

// The launch of `blocks` blocks in clusters of `size`.
struct BatchLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr = {};
    BatchLaunch(Shape shape, int blocks, int size, size_t sm, cudaStream_t st) {
        cfg.gridDim = dim3((unsigned)blocks);
        cfg.blockDim = dim3((unsigned)shape.threads);
        cfg.dynamicSmemBytes = sm;
        cfg.stream = st;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = (unsigned)size;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
};

// Clusters of `size` blocks that are resident at a time.
int resident_teams(Shape shape, int size, size_t sm, int num_sms) {
    if (size == 1) return num_sms * shape.per_sm;
    BatchLaunch l(shape, size, size, sm, nullptr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, (const void*)batch_kernel(shape), &l.cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int launch_batch(cr_context* ctx, const BatchInputs& in, const std::vector<int32_t>& order, int kmax,
                 int p, Shape shape, const TeamPlan& plan, std::vector<int32_t>* cop,
                 std::vector<cr_batch_result>* res, float* ms,
                 std::vector<unsigned long long>* times = nullptr) {
    const int count = (int)order.size();
    const int nteams = plan.resident(count), nblocks = nteams * plan.size;
    void* bufs[14] = {};
    auto cleanup = [&]() {
        for (void* q : bufs) ctx->cache.put(q);
    };
    BatchDev b;
    b.count = count;
    b.kmax = kmax;
    b.p = p;
    size_t sizes[14] = {order.size() * 4, in.n.size() * 4, in.maxdeg.size() * 4, in.rp_off.size() * 8,
                        in.col_off.size() * 8, in.rp.size() * 4, std::max<size_t>(in.col.size(), 1) * 2,
                        in.rrp.size() * 4, std::max<size_t>(in.rcol.size(), 1) * 2,
                        (size_t)nteams * plan.team_bytes, 2 * sizeof(int) + in.n.size() * 4,
                        in.n.size() * kmax * sizeof(cr_batch_result), (size_t)nblocks * 16, (size_t)nteams * sizeof(int)};
    for (int i = 0; i < 14; ++i) {
        cudaError_t e = ctx->cache.get(&bufs[i], sizes[i]);
        if (e != cudaSuccess) {
            cleanup();
            ctx->err = std::string("batch allocation: ") + cudaGetErrorString(e);
            return e == cudaErrorMemoryAllocation ? CR_ERR_NOMEM : CR_ERR_CUDA;
        }
    }
    cudaStream_t st = ctx->stream;
    const void* src[9] = {order.data(), in.n.data(), in.maxdeg.data(), in.rp_off.data(), in.col_off.data(),
                          in.rp.data(), in.col.data(), in.rrp.data(), in.rcol.data()};
    for (int i = 0; i < 9; ++i) {
        if (i == 6 && in.col.empty()) continue;
        if (i == 8 && in.rcol.empty()) continue;
        cudaMemcpyAsync(bufs[i], src[i], sizes[i], cudaMemcpyHostToDevice, st);
    }
    b.order = (const int32_t*)bufs[0];
    b.n = (const int32_t*)bufs[1];
    b.maxdeg = (const int32_t*)bufs[2];
    b.rp_off = (const uint64_t*)bufs[3];
    b.col_off = (const uint64_t*)bufs[4];
    b.rp_all = (const uint32_t*)bufs[5];
    b.col_all = (const uint16_t*)bufs[6];
    b.rrp_all = (const uint32_t*)bufs[7];
    b.rcol_all = (const uint16_t*)bufs[8];
    b.slots = (unsigned char*)bufs[9];
    b.team_bytes = plan.team_bytes;
    b.solo_bytes = plan.solo_bytes;
    b.team_count = plan.count;
    b.next = (int*)bufs[10];
    b.cop = (int32_t*)((char*)bufs[10] + 2 * sizeof(int));
    b.res = (cr_batch_result*)bufs[11];
    b.cta_time = (unsigned long long*)bufs[12];
    b.mail = (int*)bufs[13];
    const size_t sm = launch_smem(in, shape);
    b.smem_words = (uint32_t)(sm / 4);
    cudaMemsetAsync(bufs[10], 0, sizes[10], st);
    cudaMemsetAsync(bufs[11], 0, sizes[11], st);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    // the batch launch is captured once as a CUDA graph and replayed
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    raise_smem_limit((const void*)batch_kernel(shape), sm);
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        const BatchLaunch l(shape, nblocks, plan.size, sm, st);
        const cudaError_t launched = cudaLaunchKernelEx(&l.cfg, batch_kernel(shape), b);
        e = cudaStreamEndCapture(st, &graph);
        if (e == cudaSuccess) e = launched;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, graph, 0);
    if (e == cudaSuccess) {
        cudaEventRecord(e0, st);
        e = cudaGraphLaunch(exec, st);
        cudaEventRecord(e1, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) {
        cudaEventElapsedTime(ms, e0, e1);
        cop->resize(in.n.size());
        res->resize(in.n.size() * kmax);
        cudaMemcpy(cop->data(), b.cop, in.n.size() * 4, cudaMemcpyDeviceToHost);
        e = cudaMemcpy(res->data(), b.res, sizes[11], cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && times) {
            times->resize((size_t)nblocks * 2);
            e = cudaMemcpy(times->data(), b.cta_time, sizes[12], cudaMemcpyDeviceToHost);
        }
    }
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cleanup();
    if (e != cudaSuccess) {
        ctx->err = std::string("batch launch: ") + cudaGetErrorString(e);
        return CR_ERR_CUDA;
    }
    return CR_OK;
}

}  // namespace

extern "C" {

int cr_batch_solve(cr_context* ctx, const cr_graph* graphs, int32_t count, int32_t kmax, int32_t p,
                   int32_t threads_per_cta, int32_t* cop_number, cr_batch_result* results,
                   cr_batch_stats* stats) {
    if (!ctx || !graphs || count <= 0 || !cop_number || !results) return CR_ERR_INVALID;
    if (kmax < 1 || kmax > kBatchMaxK) return fail(ctx, CR_ERR_LIMIT, "batch: kmax outside 1..3");
    if (p != 1) return fail(ctx, CR_ERR_LIMIT, "batch: full visibility (p = 1) only");
    if (threads_per_cta != 0 && threads_per_cta != 256 && threads_per_cta != 512 && threads_per_cta != 1024)
        return fail(ctx, CR_ERR_INVALID, "batch: threads_per_cta must be 0 (autotune), 256, 512 or 1024");
    cudaSetDevice(ctx->device);
    BatchInputs in;
    in.n.resize(count);
    in.maxdeg.resize(count);
    in.rp_off.resize(count);
    in.col_off.resize(count);
    std::vector<double> cost(count);
    for (int i = 0; i < count; ++i) {
        const cr_graph& g = graphs[i];
        if (g.n <= 0 || g.n > kBatchMaxN || !g.row_ptr) return fail(ctx, CR_ERR_LIMIT, "batch: every graph needs 1..128 vertices");
        const uint32_t nnz = g.row_ptr[g.n];
        if (nnz && !g.col_idx) return fail(ctx, CR_ERR_INVALID, "batch: graph arrays missing");
        in.n[i] = g.n;
        in.max_n = std::max(in.max_n, g.n);
        in.rp_off[i] = in.rp.size();
        in.col_off[i] = in.col.size();
        int md = 0;
        std::vector<uint32_t> indeg(g.n + 1, 0);
        for (int v = 0; v < g.n; ++v) {
            if (g.row_ptr[v + 1] < g.row_ptr[v]) return fail(ctx, CR_ERR_INVALID, "batch: row_ptr not monotone");
            md = std::max<int>(md, g.row_ptr[v + 1] - g.row_ptr[v]);
        }
        for (uint32_t e = 0; e < nnz; ++e) {
            if (g.col_idx[e] >= g.n) return fail(ctx, CR_ERR_INVALID, "batch: neighbour index out of range");
            indeg[g.col_idx[e] + 1]++;
        }
        in.maxdeg[i] = md;
        in.max_stage_words = std::max(in.max_stage_words,
                                      and_stage_words(g.n, round_words((g.n + 31) / 32), (int)nnz));
        for (int v = 0; v <= g.n; ++v) in.rp.push_back(g.row_ptr[v]);
        for (uint32_t e = 0; e < nnz; ++e) in.col.push_back(g.col_idx[e]);
        // in-neighbour CSR (ascending sources)
        for (int v = 0; v < g.n; ++v) indeg[v + 1] += indeg[v];
        for (int v = 0; v <= g.n; ++v) in.rrp.push_back(indeg[v]);
        std::vector<uint32_t> fill(indeg.begin(), indeg.end() - 1);
        std::vector<uint16_t> rc(nnz);
        for (int u = 0; u < g.n; ++u)
            for (uint32_t e = g.row_ptr[u]; e < g.row_ptr[u + 1]; ++e) rc[fill[g.col_idx[e]]++] = (uint16_t)u;
        in.rcol.insert(in.rcol.end(), rc.begin(), rc.end());
        cost[i] = (double)binom_dev((int64_t)g.n + kmax - 1, kmax) * g.n;
    }
    std::vector<int32_t> order(count);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return cost[a] > cost[c]; });
    const size_t slot_bytes = job_layout(in.max_n, kmax, p, 2).total;

    // half of what the device has free, the context's held blocks included (an allocation that does
    // not fit otherwise gets them back)
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    const size_t memory = (free_b + ctx->cache.free_bytes()) / 2;
    auto alone = [&](Shape s) { return TeamPlan::alone(ctx->num_sms * s.per_sm, slot_bytes); };
    auto fits = [&](Shape s) { return alone(s).bytes(count) < memory; };
    Shape shape{threads_per_cta ? threads_per_cta : 512, threads_per_cta == 256 ? 2 : 1};
    if (threads_per_cta == 0) {
        // autotune: time candidate launch shapes on a calibration slice (every 8th graph of
        // the cost order, so the slice has the batch's size mix), once per device and shape
        const auto key = std::make_tuple(ctx->device, in.max_n, kmax, p);
        std::lock_guard<std::mutex> lock(g_tune_mu);
        auto it = g_tuned.find(key);
        if (it != g_tuned.end()) {
            shape = it->second;
        } else {
            std::vector<int32_t> calib;
            for (int i = 0; i < count; i += 8) calib.push_back(order[i]);
            // every shape fits the register file: 256 x 2 and 512 x 1 at 128 registers,
            // 1024 x 1 at 64
            const Shape cands[] = {{256, 2}, {512, 1}, {1024, 1}};
            float best = 1e30f;
            for (Shape c : cands) {
                if (!fits(c)) continue;
                std::vector<int32_t> cp;
                std::vector<cr_batch_result> rs;
                float ms = 0;
                if (launch_batch(ctx, in, calib, kmax, p, c, alone(c), &cp, &rs, &ms) != CR_OK) continue;
                if (ms < best) {
                    best = ms;
                    shape = c;
                }
            }
            g_tuned[key] = shape;
        }
    }
    while (!fits(shape) && shape.per_sm > 1) shape.per_sm--;
    if (!fits(shape)) return fail(ctx, CR_ERR_NOMEM, "batch: not enough device memory for one slot per SM");
    std::vector<int32_t> cop;
    std::vector<cr_batch_result> res;
    float ms = 0;
    std::vector<unsigned long long> times;
    // the teams' share of the batch
    const size_t smem = launch_smem(in, shape);
    raise_smem_limit((const void*)batch_kernel(shape), smem);
    std::vector<double> sorted(count);
    for (int i = 0; i < count; ++i) sorted[i] = cost[order[i]];
    TeamPlan plan = plan_teams(
        sorted, ctx->num_sms * shape.per_sm, slot_bytes, memory,
        [&](int size) { return resident_teams(shape, size, smem, ctx->num_sms); },
        [&](int by_teams) { return job_layout(by_teams < count ? in.n[order[by_teams]] : 1, kmax, p, 2).total; });
    int rc = launch_batch(ctx, in, order, kmax, p, shape, plan, &cop, &res, &ms, &times);
    if (rc == CR_ERR_NOMEM && plan.size > 1) {   // (taken by others meanwhile)
        cudaGetLastError();
        plan = alone(shape);
        rc = launch_batch(ctx, in, order, kmax, p, shape, plan, &cop, &res, &ms, &times);
    }
    if (rc) return rc;
    memcpy(cop_number, cop.data(), count * sizeof(int32_t));
    memcpy(results, res.data(), res.size() * sizeof(cr_batch_result));
    if (stats) {
        memset(stats, 0, sizeof(*stats));
        stats->ms = ms;
        for (const auto& r : res) stats->states += r.solved ? r.states : 0;
        stats->threads = shape.threads;
        stats->ctas = plan.resident(count) * plan.size;
        stats->slot_bytes = (int64_t)(plan.team_bytes / plan.size);
        // how evenly the blocks were kept busy: mean busy span over the whole span, and the
        // time from the median block's last graph to the last block's
        const size_t nb = times.size() / 2;
        if (nb) {
            unsigned long long t0 = ~0ull, t1 = 0;
            std::vector<double> ends(nb);
            double busy = 0;
            for (size_t i = 0; i < nb; ++i) {
                t0 = std::min(t0, times[2 * i]);
                t1 = std::max(t1, times[2 * i + 1]);
            }
            for (size_t i = 0; i < nb; ++i) {
                busy += (double)(times[2 * i + 1] - times[2 * i]);
                ends[i] = (double)(times[2 * i + 1] - t0);
            }
            std::sort(ends.begin(), ends.end());
            const double span = (double)(t1 - t0);
            stats->busy_frac = span > 0 ? busy / (span * nb) : 0;
            stats->tail_ms = (span - ends[nb / 2]) / 1e6;
        }
    }
    for (const auto& r : res)
        if (r.solved && r.status != CR_OK) return fail(ctx, CR_ERR_INTERNAL, "batch: a solve reported a device error");
    return CR_OK;
}

}  // extern "C"
