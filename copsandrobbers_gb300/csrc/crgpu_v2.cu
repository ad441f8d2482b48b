// crgpu_v2.cu - snapshot passes of the macro-turn trajectory search
// (solvers/k_cops_visibility_v2.cpp: one plane (C, r), p cop/robber steps per visibility cycle).
//
// The reference decides every unmarked (C0, r) by a branch-and-bound DFS over cop
// trajectories C1..Cp (trajectoryDFS, v2:243-341) against the table as it stood at the start
// of the pass, buffering the marks (v2:437-562).  The DFS value is the minimum, over
// trajectories, of the first event on that trajectory:
//     cop ply d empties the robber cloud          -> 2d - 1        (v2:300-308)
//     robber ply d leaves no robber alive         -> 2d            (v2:312-319)
//     d = p, cloud inside the marked set of C_p   -> 2p + max round (v2:321-334)
// Branch-and-bound order and the two skip filters (v2:450-523) change only the work, not
// that minimum, so these kernels compute it directly, level by level.
//
// Every pass needs only what the last one changed.  Terminal events do not depend on the table
// and leaves need marks besides the captures (a cloud never holds a cop), so the first pass
// evaluates terminal events only, and marks values in 1 .. 2p.  A leaf that becomes available in
// a later pass t holds a state marked in pass t - 1; by induction the marks of pass s lie in
// (2p(s-1), 2ps], so its cost lies in (2p(t-1), 2pt]: above everything found before, at any depth
// (costs are absolute plies).  Hence a node's value is final in the pass that first finds one, and
// a later pass evaluates open nodes only, from leaves at the configurations changed by the pass
// before it.  lev[j] flags the configurations with a changed one exactly j cop steps away
// (k_v2_dilate); a depth-d node has new leaves only within lev[p-d].
//
// Clouds repeat heavily.  The robber moves first, so the depth-2 node below (C1, r) with cops C2
// has the cloud N(N(r) \ C1 \ C2) \ C2: for every predecessor C1 of C2 that misses N(r) it is the
// same plain node (C2, r).  So each pass goes
//   k_v2_begin    per changed configuration C the vertices with a neighbour unmarked in row C (its
//                 unsafe row): a leaf at C is available when the cloud before the last robber ply
//                 misses them (one AND, no expansion);
//   k_v2_plain    plain[C2][r], the values of the plain depth-2 nodes;
//   k_v2_val1     val1[C1][r], the values of the depth-1 nodes (C1, N(r) \ C1): for the robbers
//                 with no cop in N(r), the minimum of the rows plain[C2] over the successors C2;
//                 for the few touched ones, child by child;
//   k_v2_root     root[C0][r] = min over C1 in T(C0) of (1 if r in C1, 2 if N(r) within C1, else
//                 val1).
//
// For p >= 3 the children of touched nodes that are not plain are deduplicated in a device hash
// table: k_v2_hinsert inserts them (key = (rank of C2 + 1) << 32 | fingerprint of the cloud,
// claimed by atomicCAS with linear probing; the claiming thread writes the full cloud beside the
// key), k_v2_heval takes the subtree minimum of each slot's node, and k_v2_val1 looks every such
// child up (key equal AND full cloud equal); a child it does not find (probe limit, table full,
// or a fingerprint shared by two clouds of the same C2, whose second cloud never got a slot) is
// evaluated directly, so the result is exact whatever the table holds.  The table is rebuilt
// every pass; when the depth-1 nodes outnumber half the table, they are processed in chunks, each
// with a fresh table.
//
// A lean solver has no plain values: every child of a depth-1 node is then looked at
// where it is reached, as a touched node's are, and three byte arrays share the memory of others
// (v2_arrays).  It serves where a memory budget or the device has no room for more; Delaunay n = 199,
// k = 2, p = 3 takes 166 ms so.
//
// Measured (Delaunay n = 199, k = 2, p = 3, six passes): 94 ms with every dirty depth-1 node's
// children in the hash table and every leaf's cloud expanded, 8.3 ms so (limits of registers were
// compared at 8.7 ms: 10.0 without one, 9.5 at 48).
#include <algorithm>
#include <string>
#include <vector>

#include "crgpu_internal.cuh"
#include "crgpu_v2.h"

namespace crgpu {

void launch_marks_from_table(const uint8_t* table, uint32_t C, int n, int cols, int rwp, uint32_t* marked,
                             int grid, cudaStream_t st);
void launch_verdict_raw(const uint8_t* table, const uint32_t* m0, uint32_t C, int n, int rw,
                        int rwp, int cols, unsigned long long* best, int grid, cudaStream_t st);

constexpr int kV2MaxP = 8;     // visibility periods handled by the device search
constexpr int kV2None = 255;   // "no winning trajectory"

struct V2Solver {
    cr_block_cache* cache = nullptr;
    cudaStream_t st = nullptr;
    int num_sms = 1;
    int n = 0, k = 0, p = 0, rw = 0, rwp = 0, W = 0;
    uint32_t C = 0;
    const uint32_t* rp = nullptr;
    const uint16_t* col = nullptr;
    const uint32_t* binom = nullptr;
    const uint16_t* configs = nullptr;
    uint8_t* table = nullptr;
    uint32_t* marked = nullptr;
    uint32_t* nbr = nullptr;
    uint8_t* val1 = nullptr;
    uint8_t* newval = nullptr;
    bool lean = false;              // without the plain values, and with shared arrays (v2_arrays)
    uint8_t* plain = nullptr;       // [C][n] plain depth-2 values; null = lean, or given back (v2_shed)
    uint32_t* unsafe = nullptr;     // [C][rwp], rows of changed configurations only
    uint8_t* changed = nullptr;     // configurations that gained marks
    uint8_t* lev = nullptr;         // [p][C]: a changed configuration j cop steps away
    uint8_t* fin1 = nullptr;        // configurations with a depth-1 / plain value found this pass
    uint8_t* fin2 = nullptr;
    uint32_t* rnbr = nullptr;       // [n][rwp]: in-neighbour masks
    uint32_t* vsets = nullptr;      // [2][rwp]: vertices with at most k moves, with none
    unsigned long long* counters = nullptr;
    unsigned int* err = nullptr;
    unsigned long long* h_pinned = nullptr;
    // depth-2 cloud table (p >= 3): key words (key and subtree value, see cloud_key) and
    // clouds [hcap][rwp]
    unsigned long long* hkey = nullptr;
    uint32_t* hmask = nullptr;
    uint64_t hcap = 0;
    uint64_t chunk_nodes = 0;   // depth-1 nodes per table fill
    cr_v2_hash_stats hstats{};
    bool first = true;
    cudaEvent_t e0 = nullptr, e1 = nullptr;   // around a pass (the solver's kit's)
    cudaEvent_t i0 = nullptr, i1 = nullptr;   // around initializeCaptures
};

struct V2Dev {
    int n, k, p, rwp;
    uint32_t C;
    const uint32_t* rp;
    const uint16_t* col;
    const uint32_t* binom;
    const uint16_t* configs;
    const uint8_t* table;
    const uint32_t* marked;
    const uint32_t* nbr;
    const uint32_t* rnbr;          // [n][rwp]: in-neighbour masks
    const uint32_t* small;         // [rwp]: vertices with at most k out-neighbours
    const uint32_t* still;         // [rwp]: vertices with none
    uint8_t* val1;
    uint8_t* newval;
    uint8_t* plain;                // null = every depth-1 node counts as touched
    uint32_t* unsafe;
    const uint8_t* lev;            // [p][C]
    uint8_t* fin1;
    uint8_t* fin2;
    bool first;                    // the first pass: terminal events only
    unsigned long long* count;     // [0] marks found, [1] depth-2 child visits, [2] table entries
    unsigned long long* hkey;      // null = no cloud table (p < 3)
    uint32_t* hmask;
    uint64_t hcap;                 // power of two
    uint64_t node_lo, node_hi;     // depth-1 nodes (C1 * n + r) of this chunk
};

constexpr int kHashProbes = 64;   // linear-probe limit of an insert or a lookup


template <int W>
struct Mask {
    uint32_t w[W];
};

template <int W>
__device__ __forceinline__ bool mask_empty(const Mask<W>& m) {
    uint32_t x = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) x |= m.w[i];
    return x == 0;
}

template <int W>
__device__ __forceinline__ uint32_t mask_word(const Mask<W>& m, int idx) {
    uint32_t x = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) x = (i == idx) ? m.w[i] : x;
    return x;
}

template <int W, int K>
__device__ __forceinline__ bool mask_hits(const Mask<W>& m, const int (&c)[K]) {
    bool hit = false;
#pragma unroll
    for (int i = 0; i < K; ++i) hit |= (mask_word<W>(m, c[i] >> 5) >> (c[i] & 31)) & 1u;
    return hit;
}

template <int W, int K>
__device__ __forceinline__ void mask_clear(Mask<W>& m, const int (&c)[K]) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
        const int wi = c[i] >> 5;
        const uint32_t b = ~(1u << (c[i] & 31));
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (j == wi) m.w[j] &= b;
    }
}

template <int W>
__device__ __forceinline__ void load_nbr(Mask<W>& m, const uint32_t* snbr, int rwp, int v) {
#pragma unroll
    for (int j = 0; j < W; ++j) m.w[j] = j < rwp ? snbr[v * rwp + j] : 0u;
}

// Robber cloud after one move: OR of the neighbour masks of every vertex of m.
template <int W>
__device__ __forceinline__ Mask<W> expand(const Mask<W>& m, const uint32_t* snbr, int rwp) {
    Mask<W> out;
#pragma unroll
    for (int j = 0; j < W; ++j) out.w[j] = 0u;
#pragma unroll
    for (int i = 0; i < W; ++i) {
        uint32_t b = m.w[i];
        while (b) {
            const int v = i * 32 + __ffs(b) - 1;
            b &= b - 1;
            const uint32_t* row = snbr + v * rwp;
#pragma unroll
            for (int j = 0; j < W; ++j)
                if (j < rwp) out.w[j] |= row[j];
        }
    }
    return out;
}

// Successor enumeration of one config: the product of each cop's neighbour list.
template <int K>
struct Moves {
    int lo[K], dg[K], T;
    int idx[K];   // odometer of the next successor tuple (last cop fastest)
};

template <int K>
__device__ __forceinline__ void moves_of(Moves<K>& mv, const int (&c)[K], const uint32_t* __restrict__ rp) {
    mv.T = 1;
#pragma unroll
    for (int i = 0; i < K; ++i) {
        mv.lo[i] = __ldg(&rp[c[i]]);
        mv.dg[i] = __ldg(&rp[c[i] + 1]) - mv.lo[i];
        mv.T *= mv.dg[i];
        mv.idx[i] = 0;
    }
}

// The successor tuple at the odometer (the same tuple move_target gives for the running
// index), then the odometer steps on: the sequential walks need no division per tuple.
template <int K>
__device__ __forceinline__ uint32_t next_target(Moves<K>& mv, const uint16_t* __restrict__ adj,
                                                const uint32_t* __restrict__ B, int np1, int (&c)[K]) {
#pragma unroll
    for (int i = 0; i < K; ++i) c[i] = __ldg(&adj[mv.lo[i] + mv.idx[i]]);
    bool carry = true;
#pragma unroll
    for (int i = K - 1; i >= 0; --i) {
        if (carry) {
            ++mv.idx[i];
            carry = mv.idx[i] >= mv.dg[i];
            if (carry) mv.idx[i] = 0;
        }
    }
    sort_small<K>(c);
    return config_rank<K>(c, B, np1);
}

template <int K>
__device__ __forceinline__ uint32_t move_target(const Moves<K>& mv, int t, const uint16_t* __restrict__ adj,
                                                const uint32_t* __restrict__ B, int np1, int (&c)[K]) {
    int rem = t;
#pragma unroll
    for (int i = K - 1; i >= 0; --i) {
        const int q = rem / mv.dg[i];
        c[i] = __ldg(&adj[mv.lo[i] + rem - q * mv.dg[i]]);
        rem = q;
    }
    sort_small<K>(c);
    return config_rank<K>(c, B, np1);
}

// Largest round among the vertices of V in row cid of the table.
template <int W>
__device__ __forceinline__ int max_round(const V2Dev& d, uint32_t cid, const Mask<W>& V) {
    const uint8_t* trow = d.table + (size_t)cid * d.n;
    int mx = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) {
        uint32_t b = V.w[i];
        while (b) {
            const int v = i * 32 + __ffs(b) - 1;
            b &= b - 1;
            mx = max(mx, (int)(__ldg(&trow[v]) >> 1));
        }
    }
    return mx;
}

// Phase D boundary (v2:321-334) for the cloud `mid` left before the last robber ply (cops c, rank
// cid): 2p + max round when its expansion lies within the marked set, which is when no vertex of
// mid has an unmarked neighbour (cops are marked in their own row), i.e. when mid misses the unsafe
// row.  Clouds whose expansion is empty are terminal and never get here.
template <int W, int K>
__device__ __forceinline__ int leaf_cost(const V2Dev& d, uint32_t cid, const int (&c)[K], const Mask<W>& mid,
                                         const uint32_t* snbr) {
    const uint32_t* urow = d.unsafe + (size_t)cid * d.rwp;
    uint32_t bad = 0u;
#pragma unroll
    for (int j = 0; j < W; ++j)
        if (j < d.rwp) bad |= mid.w[j] & __ldg(&urow[j]);
    if (bad) return kV2None;
    Mask<W> nx = expand<W>(mid, snbr, d.rwp);
    mask_clear<W, K>(nx, c);
    return 2 * d.p + max_round<W>(d, cid, nx);
}

// Whether some cop move below (c, V) can leave the robber nowhere: what a move leaves of V must
// then be vertices with at most K neighbours, and a move takes at most K vertices away.
template <int W, int K>
__device__ __forceinline__ bool may_trap(const V2Dev& d, const Mask<W>& V) {
    int big = 0;
#pragma unroll
    for (int j = 0; j < W; ++j)
        if (j < d.rwp) big += __popc(V.w[j] & ~__ldg(&d.small[j]));
    return big <= K;
}

// Minimum over the children of a depth p - 1 node (c, V).  In the first pass only the terminal
// events count (no cloud lies within the captures alone), in a later one only the leaves at
// configurations that gained marks in the last pass.
template <int W, int K>
__device__ int last_ply_min(const V2Dev& d, const int (&c)[K], const Mask<W>& V, const uint32_t* snbr, int best) {
    if (d.first && !may_trap<W, K>(d, V)) return best;
    Moves<K> mv;
    moves_of<K>(mv, c, d.rp);
    const int np1 = d.n + 1;
    for (int t = 0; t < mv.T; ++t) {
        int cp[K];
        const uint32_t cid = next_target<K>(mv, d.col, d.binom, np1, cp);
        if (cid >= d.C) continue;   // never taken for a well-formed rank table
        if (!d.first && !__ldg(&d.lev[cid])) continue;
        Mask<W> mid = V;
        mask_clear<W, K>(mid, cp);
        if (d.first) {
            if (mask_empty<W>(mid)) return min(best, 2 * d.p - 1);   // the smallest value of such a node
            Mask<W> nx = expand<W>(mid, snbr, d.rwp);
            mask_clear<W, K>(nx, cp);
            if (mask_empty<W>(nx)) best = min(best, 2 * d.p);
        } else {
            best = min(best, leaf_cost<W, K>(d, cid, cp, mid, snbr));
        }
    }
    return best;
}

template <int W, int K>
struct Frame {
    Mask<W> V, E;
    Moves<K> mv;
    int t;
};

// Minimum over the trajectory subtree below node (depth 2, cops c2, cloud V2), p >= 3, of what this
// pass can find: terminal events in the first pass, leaves at the changed configurations in the
// others, where a child at depth dc is only entered when a changed configuration lies p - dc cop
// steps away.
template <int W, int K>
__device__ int subtree_min(const V2Dev& d, const int (&c2)[K], const Mask<W>& V2, const uint32_t* snbr, int best) {
    if (d.p == 3) return last_ply_min<W, K>(d, c2, V2, snbr, best);
    Frame<W, K> st[kV2MaxP - 3];   // depths 2 .. p - 2
    int top = 0;
    st[0].V = V2;
    st[0].E = expand<W>(V2, snbr, d.rwp);
    moves_of<K>(st[0].mv, c2, d.rp);
    st[0].t = 0;
    const int np1 = d.n + 1;
    while (top >= 0) {
        Frame<W, K>& f = st[top];
        const int dc = top + 3;  // depth of the child about to be tried
        if (f.t >= f.mv.T || 2 * dc - 1 >= best) { --top; continue; }
        ++f.t;
        int c[K];
        const uint32_t cid = next_target<K>(f.mv, d.col, d.binom, np1, c);
        if (cid >= d.C) continue;
        if (!d.first && !__ldg(&d.lev[(size_t)(d.p - dc) * d.C + cid])) continue;
        Mask<W> nx;
        if (mask_hits<W, K>(f.V, c)) {
            Mask<W> mid = f.V;
            mask_clear<W, K>(mid, c);
            if (mask_empty<W>(mid)) { best = 2 * dc - 1; continue; }
            nx = expand<W>(mid, snbr, d.rwp);
        } else {
            nx = f.E;
        }
        mask_clear<W, K>(nx, c);
        if (mask_empty<W>(nx)) { best = min(best, 2 * dc); continue; }
        if (dc == d.p - 1) {
            best = last_ply_min<W, K>(d, c, nx, snbr, best);
            continue;
        }
        Frame<W, K>& g = st[top + 1];
        g.V = nx;
        g.E = expand<W>(nx, snbr, d.rwp);
        moves_of<K>(g.mv, c, d.rp);
        g.t = 0;
        ++top;
    }
    return best;
}

// Cloud-table key of depth-2 node (cid, V): the config's rank + 1 above a 24-bit fingerprint of
// the cloud, above a zero byte where the node's subtree value goes once k_v2_heval has it (one
// word per probe holds both; never 0, which marks an empty slot).
template <int W>
__device__ __forceinline__ unsigned long long cloud_key(uint32_t cid, const Mask<W>& V) {
    uint32_t h = 0x9E3779B9u;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        h = (h ^ V.w[j]) * 0x85EBCA6Bu;
        h ^= h >> 13;
    }
    h *= 0xC2B2AE35u;
    h ^= h >> 16;
    return ((unsigned long long)(cid + 1u) << 32) | ((h & 0xFFFFFFu) << 8);
}

__device__ __forceinline__ uint64_t cloud_slot(unsigned long long key, uint64_t cap) {
    uint64_t z = key + 0x9E3779B97F4A7C15ull;   // splitmix64 finaliser
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (z ^ (z >> 31)) & (cap - 1);
}

// Insert (cid, V) unless its key is present; the thread that claims a slot writes the cloud.
// Returns 1 when this call claimed a new slot.
template <int W>
__device__ __forceinline__ unsigned cloud_insert(const V2Dev& d, uint32_t cid, const Mask<W>& V) {
    const unsigned long long key = cloud_key<W>(cid, V);
    uint64_t h = cloud_slot(key, d.hcap);
    for (int probe = 0; probe < kHashProbes; ++probe) {
        const unsigned long long old = atomicCAS(&d.hkey[h], 0ull, key);
        if (old == 0ull) {
            uint32_t* m = d.hmask + h * d.rwp;
#pragma unroll
            for (int j = 0; j < W; ++j)
                if (j < d.rwp) m[j] = V.w[j];
            return 1u;
        }
        if (old == key) return 0u;
        h = (h + 1) & (d.hcap - 1);
    }
    return 0u;   // probe limit: the lookup misses and the node is evaluated directly
}

// Stored value of (cid, V), or -1 when the table does not hold exactly this node.
template <int W>
__device__ __forceinline__ int cloud_lookup(const V2Dev& d, uint32_t cid, const Mask<W>& V) {
    const unsigned long long key = cloud_key<W>(cid, V);
    uint64_t h = cloud_slot(key, d.hcap);
    for (int probe = 0; probe < kHashProbes; ++probe) {
        const unsigned long long k = __ldg(&d.hkey[h]);
        if (k == 0ull) return -1;
        if ((k & ~0xFFull) == key) {
            const uint32_t* m = d.hmask + h * d.rwp;
            bool same = true;
#pragma unroll
            for (int j = 0; j < W; ++j)
                if (j < d.rwp) same &= __ldg(&m[j]) == V.w[j];
            return same ? (int)(k & 0xFFull) : -1;
        }
        h = (h + 1) & (d.hcap - 1);
    }
    return -1;
}

template <int K>
__device__ __forceinline__ void cops_of(const V2Dev& d, uint32_t cid, int (&c)[K]) {
#pragma unroll
    for (int i = 0; i < K; ++i) c[i] = d.configs[(size_t)cid * K + i];
}

// The robbers r whose neighbourhood one of the cops stands in (N(r) meets C), cops left out: their
// depth-1 clouds N(r) \ C are not N(r) itself.  Without plain values: all but the cops.
template <int W, int K>
__device__ __forceinline__ Mask<W> touched_robbers(const V2Dev& d, const int (&c)[K]) {
    Mask<W> e;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        e.w[j] = d.plain ? 0u : valid_mask(d.n, j);
        if (j < d.rwp)
#pragma unroll
            for (int i = 0; i < K; ++i) e.w[j] |= __ldg(&d.rnbr[c[i] * d.rwp + j]);
    }
    mask_clear<W, K>(e, c);
    return e;
}

// The child (C2, r) of a touched depth-1 node is the plain one of k_v2_plain when every cop of C1
// in N(r) stands on a vertex of C2 too: C1 then takes nothing from N(r) that C2 does not.
template <int W, int K>
__device__ __forceinline__ bool plain_child(const Mask<W>& nr, const int (&c1)[K], const int (&c2)[K]) {
    bool plain = true;
#pragma unroll
    for (int i = 0; i < K; ++i) {
        bool in = false;
#pragma unroll
        for (int j = 0; j < K; ++j) in |= c1[i] == c2[j];
        plain &= in || !((mask_word<W>(nr, c1[i] >> 5) >> (c1[i] & 31)) & 1u);
    }
    return plain;
}

__device__ __forceinline__ void load_graph(const V2Dev& d, uint32_t* snbr) {
    for (int i = threadIdx.x; i < d.n * d.rwp; i += blockDim.x) snbr[i] = d.nbr[i];
    __syncthreads();
}

// The begin of a pass after the first (whose clears are k_v2_init's), a warp per configuration: the
// counters and the flags of what this pass finds are cleared, the last pass's changes become lev[0],
// and a changed configuration gets its unsafe row (a lane per vertex): bit v of row C set iff v has a
// neighbour unmarked in row C.
template <int W>
__global__ void __launch_bounds__(256) k_v2_begin(V2Dev d, uint8_t* lev0, uint8_t* changed) {
    extern __shared__ uint32_t snbr[];
    load_graph(d, snbr);
    if (blockIdx.x == 0 && threadIdx.x < 3) d.count[threadIdx.x] = 0ull;
    const int lane = threadIdx.x & 31;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < d.C; c += nwarps) {
        const uint8_t ch = changed[c];
        __syncwarp();
        if (lane == 0) {
            if (lev0 != changed) {
                lev0[c] = ch;
                changed[c] = 0;
            }
            d.fin1[c] = 0;
            d.fin2[c] = 0;
        }
        if (!ch) continue;
        Mask<W> m;
#pragma unroll
        for (int j = 0; j < W; ++j) m.w[j] = j < d.rwp ? __ldg(&d.marked[(size_t)c * d.rwp + j]) : 0u;
        for (int w = 0; w < d.rwp; ++w) {
            const int v = w * 32 + lane;
            uint32_t out = 0u;
            if (v < d.n) {
#pragma unroll
                for (int j = 0; j < W; ++j)
                    if (j < d.rwp) out |= snbr[v * d.rwp + j] & ~m.w[j];
            }
            const unsigned u = __ballot_sync(0xFFFFFFFFu, out != 0u);
            if (lane == 0) d.unsafe[(size_t)c * d.rwp + w] = u;
        }
    }
}

// Values of the plain depth-2 nodes plain[C2][r]: cloud N(N(r) \ C2) \ C2, the child of every
// depth-1 node (C1, r) whose cops miss N(r).  3 / 4 = the cloud is empty after the cops' or the
// robber's second ply; else p = 2: the leaf's cost; p >= 3: the subtree minimum.  A warp per
// configuration C2, a lane per robber; for p = 3 the warp walks the moves in step (the changed
// ones of 32 at a time), so a leaf test is one unsafe row, the same for all lanes, ANDed with each
// lane's cloud.  Values are final once found (see the head of this file): later passes look at
// the open nodes only.
template <int K, int W>
__global__ void __launch_bounds__(256, 4) k_v2_plain(V2Dev d) {
    extern __shared__ uint32_t snbr[];
    load_graph(d, snbr);
    const int lane = threadIdx.x & 31;
    const int np1 = d.n + 1;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t c2 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c2 < d.C; c2 += nwarps) {
        if (!d.first && !d.lev[(size_t)(d.p - 2) * d.C + c2]) continue;
        int cops[K];
        cops_of<K>(d, c2, cops);
        Moves<K> mv;
        moves_of<K>(mv, cops, d.rp);
        bool found = false;
        for (int rb = 0; rb < d.n; rb += 32) {
            const int r = rb + lane;
            const size_t at = (size_t)c2 * d.n + r;
            bool open = r < d.n && (d.first || d.plain[at] == kV2None);
            if (!__any_sync(0xFFFFFFFFu, open)) continue;
            int val = kV2None;
            Mask<W> mid, V;
            load_nbr<W>(mid, snbr, d.rwp, open ? r : 0);
            mask_clear<W, K>(mid, cops);
            V = expand<W>(mid, snbr, d.rwp);
            mask_clear<W, K>(V, cops);
            if (d.first) {
                if (mask_empty<W>(mid)) val = 3;
                else if (mask_empty<W>(V)) val = 4;
            }
            if (open && val == kV2None) {
                if (d.p == 2) {
                    if (!d.first) val = leaf_cost<W, K>(d, c2, cops, mid, snbr);
                } else if (d.first || d.p > 3) {
                    val = subtree_min<W, K>(d, cops, V, snbr, kV2None);
                }
            }
            if (d.p == 3 && !d.first) {
                for (int t0 = 0; t0 < mv.T; t0 += 32) {
                    int c3[K];
                    uint32_t cid = 0;
                    bool go = false;
                    if (t0 + lane < mv.T) {
                        cid = move_target<K>(mv, t0 + lane, d.col, d.binom, np1, c3);
                        go = cid < d.C && d.lev[cid];
                    }
                    unsigned todo = __ballot_sync(0xFFFFFFFFu, go);
                    while (todo) {
                        const int b = __ffs(todo) - 1;
                        todo &= todo - 1;
                        const uint32_t id = __shfl_sync(0xFFFFFFFFu, cid, b);
                        int c[K];
#pragma unroll
                        for (int i = 0; i < K; ++i) c[i] = __shfl_sync(0xFFFFFFFFu, c3[i], b);
                        if (open) {
                            Mask<W> m = V;
                            mask_clear<W, K>(m, c);
                            val = min(val, leaf_cost<W, K>(d, id, c, m, snbr));
                        }
                    }
                }
            }
            if (open && (d.first || val != kV2None)) {
                d.plain[at] = (uint8_t)min(val, kV2None);
                found |= val != kV2None;
            }
        }
        if (__any_sync(0xFFFFFFFFu, found) && lane == 0) d.fin2[c2] = 1;
    }
}

// Fill the cloud table with the distinct non-terminal depth-2 children of the chunk's touched
// depth-1 nodes that are still open, plain ones (k_v2_plain) left out: a warp per configuration,
// its touched robbers one by one, lanes over the cop moves.
template <int K, int W>
__global__ void __launch_bounds__(256, 4) k_v2_hinsert(V2Dev d) {
    extern __shared__ uint32_t snbr[];
    load_graph(d, snbr);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const int np1 = d.n + 1;
    const uint32_t c_hi = (uint32_t)((d.node_hi + d.n - 1) / d.n);
    unsigned visits = 0, fresh = 0;
    for (uint32_t c1 = (uint32_t)(d.node_lo / d.n) + blockIdx.x * (blockDim.x >> 5) + warp; c1 < c_hi; c1 += nwarps) {
        if (!d.first && !d.lev[(size_t)(d.p - 1) * d.C + c1]) continue;
        int cops1[K];
        cops_of<K>(d, c1, cops1);
        const Mask<W> touched = touched_robbers<W, K>(d, cops1);
        Moves<K> mv;
        moves_of<K>(mv, cops1, d.rp);
        for (int j = 0; j < d.rwp; ++j) {
            uint32_t bits = mask_word<W>(touched, j);
            while (bits) {
                const int r = j * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
                const size_t idx = (size_t)c1 * d.n + r;
                if (idx < d.node_lo || idx >= d.node_hi || (!d.first && d.val1[idx] != kV2None)) continue;
                Mask<W> nr, V1;
                load_nbr<W>(nr, snbr, d.rwp, r);
                V1 = nr;
                mask_clear<W, K>(V1, cops1);
                if (mask_empty<W>(V1)) continue;
                for (int t = lane; t < mv.T; t += 32) {
                    int c2[K];
                    const uint32_t cid2 = move_target<K>(mv, t, d.col, d.binom, np1, c2);
                    if (cid2 >= d.C || (!d.first && !d.lev[(size_t)(d.p - 2) * d.C + cid2])) continue;
                    if (d.plain && plain_child<W, K>(nr, cops1, c2)) continue;
                    Mask<W> mid = V1;
                    mask_clear<W, K>(mid, c2);
                    if (mask_empty<W>(mid)) continue;
                    Mask<W> nx = expand<W>(mid, snbr, d.rwp);
                    mask_clear<W, K>(nx, c2);
                    if (mask_empty<W>(nx)) continue;
                    ++visits;
                    fresh += cloud_insert<W>(d, cid2, nx);
                }
            }
        }
    }
    visits = __reduce_add_sync(0xFFFFFFFFu, visits);
    fresh = __reduce_add_sync(0xFFFFFFFFu, fresh);
    if (lane == 0) {
        if (visits) atomicAdd(&d.count[1], (unsigned long long)visits);
        if (fresh) atomicAdd(&d.count[2], (unsigned long long)fresh);
    }
}

// Subtree minimum of every node in the cloud table.  Few of the slots are taken (one in ten on a
// Delaunay graph of 199 vertices), so each warp gathers the taken ones of its stretch in shared
// memory and evaluates 32 at a time, a lane each: 1.70 ms a thread per slot, 0.61 ms so (largest pass of that solve).
template <int K, int W>
__global__ void __launch_bounds__(256, 4) k_v2_heval(V2Dev d) {
    extern __shared__ uint32_t snbr[];
    __shared__ uint64_t s_slots[8][64];
    load_graph(d, snbr);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint64_t* slots = s_slots[warp];
    int held = 0;   // warp-uniform
    const uint64_t nwarps = (uint64_t)gridDim.x * 8;
    const uint64_t per = (d.hcap / 32 + nwarps - 1) / nwarps * 32;   // (the capacity is a multiple of 1024)
    const uint64_t lo = ((uint64_t)blockIdx.x * 8 + warp) * per, hi = lo + per < d.hcap ? lo + per : d.hcap;
    for (uint64_t h0 = lo; h0 < hi || held > 0; h0 += 32) {
        if (h0 < hi) {
            const bool taken = d.hkey[h0 + lane] != 0ull;
            const unsigned b = __ballot_sync(0xFFFFFFFFu, taken);
            if (taken) slots[held + __popc(b & ((1u << lane) - 1u))] = h0 + lane;
            held += __popc(b);
            __syncwarp();
            if (held < 32 && h0 + 32 < hi) continue;
        }
        const int take = min(held, 32);
        if (lane < take) {
            const uint64_t h = slots[lane];
            const unsigned long long key = d.hkey[h];
            const uint32_t cid = (uint32_t)(key >> 32) - 1u;
            int c2[K];
            cops_of<K>(d, cid, c2);
            Mask<W> V;
#pragma unroll
            for (int j = 0; j < W; ++j) V.w[j] = j < d.rwp ? d.hmask[h * d.rwp + j] : 0u;
            const int v = subtree_min<W, K>(d, c2, V, snbr, kV2None);
            d.hkey[h] = key | (unsigned long long)min(v, kV2None);   // the value in the key word's low byte
        }
        __syncwarp();
        uint64_t rest = 0;
        if (lane + 32 < held) rest = slots[lane + 32];
        __syncwarp();
        if (lane + 32 < held) slots[lane] = rest;
        held -= take;
        __syncwarp();
    }
}

// Depth-1 values: a warp per configuration C1 of the chunk.  The robbers whose neighbourhood no
// cop of C1 stands in, a lane each: the minimum of plain[C2][r] over the successors C2 (whole rows
// of bytes, the same C2 for all lanes; in later passes only the C2 that found something).  Then
// the touched robbers one by one, lanes over the successors: a plain child's value, or the cloud
// table's, or the node evaluated in place.
template <int K, int W>
__global__ void __launch_bounds__(256, 4) k_v2_val1(V2Dev d) {
    extern __shared__ uint32_t snbr[];
    load_graph(d, snbr);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const int np1 = d.n + 1;
    const uint32_t c_hi = (uint32_t)((d.node_hi + d.n - 1) / d.n);
    unsigned visits = 0;
    for (uint32_t c1 = (uint32_t)(d.node_lo / d.n) + blockIdx.x * (blockDim.x >> 5) + warp; c1 < c_hi; c1 += nwarps) {
        if (!d.first && !d.lev[(size_t)(d.p - 1) * d.C + c1]) continue;
        int cops1[K];
        cops_of<K>(d, c1, cops1);
        bool found = false;
        if (d.p == 1) {   // the depth-1 nodes are the leaves
            if (!d.first) {
                for (int r = lane; r < d.n; r += 32) {
                    const size_t idx = (size_t)c1 * d.n + r;
                    if (idx < d.node_lo || idx >= d.node_hi || d.val1[idx] != kV2None) continue;
                    bool rin = false;
#pragma unroll
                    for (int i = 0; i < K; ++i) rin |= cops1[i] == r;
                    if (rin || ((d.unsafe[(size_t)c1 * d.rwp + (r >> 5)] >> (r & 31)) & 1u)) continue;
                    Mask<W> V1;
                    load_nbr<W>(V1, snbr, d.rwp, r);
                    mask_clear<W, K>(V1, cops1);
                    if (mask_empty<W>(V1)) continue;
                    d.val1[idx] = (uint8_t)(2 + max_round<W>(d, c1, V1));
                    found = true;
                }
            }
            if (__any_sync(0xFFFFFFFFu, found) && lane == 0) d.fin1[c1] = 1;
            continue;
        }
        const Mask<W> touched = touched_robbers<W, K>(d, cops1);
        Moves<K> mv;
        moves_of<K>(mv, cops1, d.rp);
        for (int rb = 0; rb < d.n; rb += 32) {
            const int r = rb + lane;
            const size_t idx = (size_t)c1 * d.n + r;
            bool open = r < d.n && idx >= d.node_lo && idx < d.node_hi;
            open = open && !((mask_word<W>(touched, r >> 5) >> (r & 31)) & 1u) && !((__ldg(&d.still[r >> 5]) >> (r & 31)) & 1u);
#pragma unroll
            for (int i = 0; i < K; ++i) open = open && cops1[i] != r;
            if (open && !d.first) open = d.val1[idx] == kV2None;
            if (!__any_sync(0xFFFFFFFFu, open)) continue;
            int best = kV2None;
            for (int t0 = 0; t0 < mv.T; t0 += 32) {
                int c2[K];
                uint32_t cid = 0;
                bool go = false;
                if (t0 + lane < mv.T) {
                    cid = move_target<K>(mv, t0 + lane, d.col, d.binom, np1, c2);
                    go = cid < d.C && d.fin2[cid];
                    if (d.first) go = cid < d.C;
                }
                unsigned todo = __ballot_sync(0xFFFFFFFFu, go);
                while (todo) {
                    const uint32_t id = __shfl_sync(0xFFFFFFFFu, cid, __ffs(todo) - 1);
                    todo &= todo - 1;
                    if (open) {
                        const int v = d.plain[(size_t)id * d.n + r];
                        best = min(best, v);
                        visits += v > 4;
                    }
                }
            }
            if (open && best < kV2None) {
                d.val1[idx] = (uint8_t)best;
                found = true;
            }
        }
        for (int j = 0; j < d.rwp; ++j) {
            uint32_t bits = mask_word<W>(touched, j);
            while (bits) {
                const int r = j * 32 + __ffs(bits) - 1;
                bits &= bits - 1;
                const size_t idx = (size_t)c1 * d.n + r;
                if (idx < d.node_lo || idx >= d.node_hi || (!d.first && d.val1[idx] != kV2None)) continue;
                Mask<W> nr, V1;
                load_nbr<W>(nr, snbr, d.rwp, r);
                V1 = nr;
                mask_clear<W, K>(V1, cops1);
                if (mask_empty<W>(V1)) continue;
                int best = kV2None;
                for (int t = lane; t < mv.T; t += 32) {
                    int c2[K];
                    const uint32_t cid2 = move_target<K>(mv, t, d.col, d.binom, np1, c2);
                    if (cid2 >= d.C || (!d.first && !d.lev[(size_t)(d.p - 2) * d.C + cid2])) continue;
                    if (d.plain && plain_child<W, K>(nr, cops1, c2)) {
                        best = min(best, (int)d.plain[(size_t)cid2 * d.n + r]);
                        continue;
                    }
                    Mask<W> mid = V1;
                    mask_clear<W, K>(mid, c2);
                    if (mask_empty<W>(mid)) { best = min(best, 3); continue; }
                    if (d.p == 2 && !d.first) {
                        best = min(best, leaf_cost<W, K>(d, cid2, c2, mid, snbr));
                        continue;
                    }
                    Mask<W> nx = expand<W>(mid, snbr, d.rwp);
                    mask_clear<W, K>(nx, c2);
                    if (mask_empty<W>(nx)) { best = min(best, 4); continue; }
                    if (d.p == 2 || best <= 5) continue;
                    // the cloud table holds the node unless an insert gave up on it
                    const int v = d.hkey ? cloud_lookup<W>(d, cid2, nx) : -1;
                    best = v >= 0 ? min(best, v) : subtree_min<W, K>(d, c2, nx, snbr, best);
                }
                best = __reduce_min_sync(0xFFFFFFFFu, best);
                if (best < kV2None) {
                    if (lane == 0) d.val1[idx] = (uint8_t)best;
                    found = true;
                }
            }
        }
        if (__any_sync(0xFFFFFFFFu, found) && lane == 0) d.fin1[c1] = 1;
    }
    visits = __reduce_add_sync(0xFFFFFFFFu, visits);
    if (lane == 0 && visits) atomicAdd(&d.count[1], (unsigned long long)visits);
}

// Root values of the unmarked states; buffered in newval (the snapshot stays intact).  A warp per
// configuration, a lane per robber, the successors 32 at a time; in later passes only the
// successors that found something (a state unmarked so far has no older value).
template <int K, int W>
__global__ void __launch_bounds__(256) k_v2_root(V2Dev d) {
    extern __shared__ uint32_t snbr[];
    if (d.first) load_graph(d, snbr);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const int np1 = d.n + 1;
    unsigned cnt = 0;
    for (uint32_t c0 = blockIdx.x * (blockDim.x >> 5) + warp; c0 < d.C; c0 += nwarps) {
        const uint32_t* mrow = d.marked + (size_t)c0 * d.rwp;
        int cops0[K];
        cops_of<K>(d, c0, cops0);
        Moves<K> mv;
        moves_of<K>(mv, cops0, d.rp);
        if (!d.first) {   // nothing found below: the common case
            bool any = false;
            for (int t = lane; t < mv.T; t += 32) {
                int c1[K];
                const uint32_t cid = move_target<K>(mv, t, d.col, d.binom, np1, c1);
                any |= cid < d.C && d.fin1[cid];
            }
            if (!__any_sync(0xFFFFFFFFu, any)) continue;
        }
        for (int rb = 0; rb < d.n; rb += 32) {
            const int r = rb + lane;
            const bool live = r < d.n && !((__ldg(&mrow[r >> 5]) >> (r & 31)) & 1u);
            if (!__any_sync(0xFFFFFFFFu, live)) continue;
            int best = kV2None;
            Mask<W> nr;
            // cop ply 1 catches r, or leaves it no move: only robbers with at most K moves
            const bool few = d.first && live && ((__ldg(&d.small[r >> 5]) >> (r & 31)) & 1u);
            if (few) load_nbr<W>(nr, snbr, d.rwp, r);
            for (int t0 = 0; t0 < mv.T; t0 += 32) {
                int own[K];
                uint32_t cid = 0;
                bool go = false;
#pragma unroll
                for (int i = 0; i < K; ++i) own[i] = 0;
                if (t0 + lane < mv.T) {
                    cid = move_target<K>(mv, t0 + lane, d.col, d.binom, np1, own);
                    go = cid < d.C && (d.first || d.fin1[cid]);
                }
                unsigned todo = __ballot_sync(0xFFFFFFFFu, go);
                while (todo) {
                    const int b = __ffs(todo) - 1;
                    todo &= todo - 1;
                    const uint32_t id = __shfl_sync(0xFFFFFFFFu, cid, b);
                    if (d.first) {
                        int c1[K];
                        bool rin = false;
#pragma unroll
                        for (int i = 0; i < K; ++i) {
                            c1[i] = __shfl_sync(0xFFFFFFFFu, own[i], b);
                            rin |= c1[i] == r;
                        }
                        if (rin) {
                            best = 1;
                        } else if (few) {
                            Mask<W> v1 = nr;
                            mask_clear<W, K>(v1, c1);
                            if (mask_empty<W>(v1)) best = min(best, 2);
                        }
                    }
                    if (live) best = min(best, (int)d.val1[(size_t)id * d.n + r]);
                }
            }
            if (live && best < kMaxRound) {
                d.newval[(size_t)c0 * d.n + r] = (uint8_t)best;
                ++cnt;
            }
        }
    }
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    if (lane == 0 && cnt) atomicAdd(d.count, (unsigned long long)cnt);
}

// Apply the buffered marks (v2:541-557).  The pass's three counts, final by now, go to the host's pinned
// words from here: a copy of its own cost a pass of the smallest solves 4 us.
__global__ void k_v2_apply(uint8_t* table, uint32_t* marked, uint8_t* newval, uint8_t* changed,
                           uint32_t C, int n, int rwp, const unsigned long long* count,
                           volatile unsigned long long* out) {
    if (blockIdx.x == 0 && threadIdx.x < 3) out[threadIdx.x] = count[threadIdx.x];
    const size_t total = (size_t)C * n;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        const uint8_t v = newval[i];
        if (v == kV2None) continue;
        newval[i] = kV2None;
        table[i] = (uint8_t)(1 | (v << 1));
        const uint32_t c = (uint32_t)(i / n);
        const int r = (int)(i - (size_t)c * n);
        atomicOr(&marked[(size_t)c * rwp + (r >> 5)], 1u << (r & 31));
        changed[c] = 1;
    }
}

// initializeCaptures over a table of unmarked bytes: the captures' bytes and the marked rows, written
// whole, and what the first pass begins with: counters and flags cleared (no configuration counts as
// changed, leaves at captures alone are never available).
__global__ void k_v2_init(uint8_t* table, uint32_t* marked, uint8_t* changed, uint8_t* fin1, uint8_t* fin2,
                          unsigned long long* count, const uint16_t* configs, uint32_t C, int n, int k, int rwp) {
    if (blockIdx.x == 0 && threadIdx.x < 3) count[threadIdx.x] = 0ull;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
        changed[c] = 0;
        fin1[c] = 0;
        fin2[c] = 0;
        for (int w = 0; w < rwp; ++w) marked[(size_t)c * rwp + w] = 0u;
        int prev = -1;
        for (int i = 0; i < k; ++i) {
            const int r = configs[(size_t)c * k + i];
            if (r == prev) continue;
            prev = r;
            table[(size_t)c * n + r] = 1;
            marked[(size_t)c * rwp + (r >> 5)] |= 1u << (r & 31);
        }
    }
}

// out[C] = OR over C' in T(C) of in[C']  (one cop step of the dirty-region dilation).
template <int K>
__global__ void k_v2_dilate(const uint8_t* __restrict__ in, uint8_t* out, const uint16_t* configs,
                            uint32_t C, int n, const uint32_t* rp, const uint16_t* adj,
                            const uint32_t* B) {
    const int np1 = n + 1;
    for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < C; c += gridDim.x * blockDim.x) {
        int cops[K];
#pragma unroll
        for (int i = 0; i < K; ++i) cops[i] = configs[(size_t)c * K + i];
        Moves<K> mv;
        moves_of<K>(mv, cops, rp);
        uint8_t any = 0;
        for (int t = 0; t < mv.T && !any; ++t) {
            int cc[K];
            const uint32_t s = next_target<K>(mv, adj, B, np1, cc);
            any = s < C ? in[s] : 0;
        }
        out[c] = any ? 1 : 0;
    }
}

// ------------------------------------------------------------------------------ host ---

// Slots of the depth-2 cloud table: twice the depth-1 nodes (about 1.2 distinct children per
// node on the graphs measured), a power of two between 2^10 and 2^24; 0 below p = 3.
static uint64_t v2_hash_capacity(uint64_t nodes, int p) {
    if (p < 3) return 0;
    uint64_t cap = 1024;
    while (cap < 2 * nodes && cap < (1ull << 24)) cap <<= 1;
    return cap;
}

uint64_t v2_footprint(int n, int k, int p) {
    long double C = 1;
    for (int i = 1; i <= k; ++i) C = C * (n + k - i) / i;
    const uint64_t c = (uint64_t)C;
    const int rwp = round_words((n + 31) / 32);
    const uint64_t hcap = v2_hash_capacity(c * (uint64_t)n, p);
    return c * n * 4 + 2 * c * (uint64_t)rwp * 4 + c * (3 + kV2MaxP) + 2 * (uint64_t)n * rwp * 4 + c * (uint64_t)k * 2 +
           hcap * (8 + 4 * (uint64_t)rwp) + (1u << 16);
}

// Of a lean solver (see v2_arrays): at most half of that, so much less that the table makes room for the
// levels beyond the second (0 = none; a table of the least size stays).  A lean solver then holds no
// more than three bytes a state, three a configuration, the marks and a table of the usual size.
static uint64_t v2_lean_hash_capacity(uint64_t C, int n, int p, int rwp) {
    const uint64_t full = v2_hash_capacity(C * n, p), slot = 8 + 4 * (uint64_t)rwp;
    if (full <= 1024) return full;
    uint64_t cap = full / 2;
    while (cap && (full - cap) * slot < C * (uint64_t)(p - 2)) cap = cap > 1024 ? cap / 2 : 0;
    return cap;
}

uint64_t v2_lean_footprint(int n, int k, int p) {
    long double C = 1;
    for (int i = 1; i <= k; ++i) C = C * (n + k - i) / i;
    const uint64_t c = (uint64_t)C;
    const int rwp = round_words((n + 31) / 32);
    const uint64_t hcap = v2_lean_hash_capacity(c, n, p, rwp);
    return c * n * 3 + c * (uint64_t)rwp * 4 + c * (1 + (uint64_t)p) + (uint64_t)n * rwp * 4 + c * (uint64_t)k * 2 +
           hcap * (8 + 4 * (uint64_t)rwp) + (60u << 10);
}

static int v2_w(int rwp) { return rwp <= 1 ? 1 : rwp <= 2 ? 2 : rwp <= 4 ? 4 : rwp <= 8 ? 8 : 16; }

static V2Dev v2_view(const V2Solver* s) {
    V2Dev d;
    d.n = s->n; d.k = s->k; d.p = s->p; d.rwp = s->rwp; d.C = s->C;
    d.rp = s->rp; d.col = s->col; d.binom = s->binom; d.configs = s->configs;
    d.table = s->table; d.marked = s->marked; d.nbr = s->nbr;
    d.val1 = s->val1; d.newval = s->newval; d.count = s->counters;
    d.plain = s->plain; d.unsafe = s->unsafe; d.lev = s->lev; d.fin1 = s->fin1; d.fin2 = s->fin2;
    d.rnbr = s->rnbr; d.small = s->vsets; d.still = s->vsets + s->rwp;
    d.first = s->first;
    d.hkey = s->hkey; d.hmask = s->hmask; d.hcap = s->hcap;
    d.node_lo = 0;
    d.node_hi = (uint64_t)s->C * s->n;
    return d;
}

#define V2_CUDA(call)                                                                     \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            if (err) *err = std::string(#call) + ": " + cudaGetErrorString(e_);          \
            return e_ == cudaErrorMemoryAllocation ? CR_ERR_NOMEM : CR_ERR_CUDA;          \
        }                                                                                 \
    } while (0)

int v2_set_hash_capacity(V2Solver* s, uint64_t slots, std::string* err) {
    if (s->p < 3) slots = 0;
    uint64_t cap = 0;
    if (slots) {
        if (slots > (1ull << 40)) {
            if (err) *err = "v2 cloud table: at most 2^40 slots";
            return CR_ERR_LIMIT;
        }
        cap = 1024;
        while (cap < slots) cap <<= 1;
    }
    V2_CUDA(cudaStreamSynchronize(s->st));
    void* old[] = {s->hkey, s->hmask};
    for (void* q : old)
        s->cache->put(q);
    s->hkey = nullptr;
    s->hmask = nullptr;
    s->hcap = 0;
    s->chunk_nodes = 0;
    s->hstats.capacity = 0;
    if (!cap) return CR_OK;
    // a solver whose table could not be allocated keeps working without one (every depth-2
    // node evaluated where it is reached)
    cudaError_t e = s->cache->get((void**)&s->hkey, cap * sizeof(unsigned long long));
    if (e == cudaSuccess) e = s->cache->get((void**)&s->hmask, cap * s->rwp * sizeof(uint32_t));
    if (e != cudaSuccess) {
        void* got[] = {s->hkey, s->hmask};
        for (void* q : got)
            s->cache->put(q);
        s->hkey = nullptr;
        s->hmask = nullptr;
        if (err) *err = std::string("v2 cloud table: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? CR_ERR_NOMEM : CR_ERR_CUDA;
    }
    s->hcap = cap;
    s->chunk_nodes = cap / 2;
    s->hstats.capacity = cap;
    return CR_OK;
}

static void v2_put_arrays(V2Solver* s) {
    if (s->unsafe == (void*)s->newval) s->unsafe = nullptr;   // (a lean solver's shared arrays)
    if (s->changed == s->lev) s->changed = nullptr;
    if (s->fin2 == s->fin1) s->fin2 = nullptr;
    void* ptrs[] = {s->plain, s->unsafe, s->changed, s->lev, s->fin1, s->fin2, s->hkey, s->hmask};
    for (void* q : ptrs) s->cache->put(q);
    s->plain = s->changed = s->lev = s->fin1 = s->fin2 = nullptr;
    s->unsafe = s->hmask = nullptr;
    s->hkey = nullptr;
}

// The arrays that a lean solver has fewer of.  There the unsafe rows, which k_v2_root does not need, lie
// in newval, which only it and k_v2_apply do; the changed flags are lev[0] itself, which nothing needs
// once k_v2_apply sets new ones (v2_pass clears both in between); no kernel sets or takes fin2.
static int v2_arrays(V2Solver* s, bool lean, std::string* err) {
    v2_put_arrays(s);
    s->lean = lean;
    const size_t C = s->C, n = s->n;
    V2_CUDA(s->cache->get((void**)&s->lev, C * s->p));
    V2_CUDA(s->cache->get((void**)&s->fin1, C));
    if (lean && (size_t)s->rwp * 4 <= n) s->unsafe = reinterpret_cast<uint32_t*>(s->newval);
    else V2_CUDA(s->cache->get((void**)&s->unsafe, C * s->rwp * 4));   // (lean: below 4 vertices)
    if (lean) {
        s->changed = s->lev;
        s->fin2 = s->fin1;
    } else {
        V2_CUDA(s->cache->get((void**)&s->plain, C * n));
        V2_CUDA(s->cache->get((void**)&s->changed, C));
        V2_CUDA(s->cache->get((void**)&s->fin2, C));
    }
    const uint64_t slots = lean ? v2_lean_hash_capacity(C, s->n, s->p, s->rwp) : v2_hash_capacity(C * n, s->p);
    return v2_set_hash_capacity(s, slots, err);
}

// Between passes: from here on every depth-1 node counts as touched, whose open children the passes look
// at where they are reached (what the plain values had found has already reached the nodes above).
bool v2_shed(V2Solver* s) {
    if (!s->plain) return false;
    s->cache->put(s->plain);
    s->plain = nullptr;
    return true;
}

int v2_create(V2Solver** out, cr_block_cache* cache, const cr_solver_kit& kit, cudaStream_t st, int num_sms, int n, int k, int p,
              const uint32_t* d_rp, const uint16_t* d_col, const uint32_t* h_rp,
              const uint16_t* h_col, const uint32_t* d_binom, const uint16_t* d_configs,
              uint32_t C, bool lean, std::string* err) {
    if (n > 512) {
        if (err) *err = "v2 rules: clouds are limited to 512 vertices";
        return CR_ERR_LIMIT;
    }
    if (p > kV2MaxP) {
        if (err) *err = "v2 rules: visibility period limited to 8";
        return CR_ERR_LIMIT;
    }
    V2Solver* s = new V2Solver();
    *out = s;
    s->cache = cache;
    s->h_pinned = kit.pinned;
    s->e0 = kit.ev[0];
    s->e1 = kit.ev[1];
    s->i0 = kit.ev[2];
    s->i1 = kit.ev[3];
    s->st = st; s->num_sms = num_sms; s->n = n; s->k = k; s->p = p; s->C = C;
    s->rw = (n + 31) / 32;
    s->rwp = round_words(s->rw);
    s->W = v2_w(s->rwp);
    s->rp = d_rp; s->col = d_col; s->binom = d_binom; s->configs = d_configs;
    V2_CUDA(s->cache->get((void**)&s->table, (size_t)C * n));
    V2_CUDA(s->cache->get((void**)&s->marked, (size_t)C * s->rwp * 4));
    V2_CUDA(s->cache->get((void**)&s->nbr, (size_t)n * s->rwp * 4));
    V2_CUDA(s->cache->get((void**)&s->val1, (size_t)C * n));
    V2_CUDA(s->cache->get((void**)&s->newval, (size_t)C * n));
    V2_CUDA(s->cache->get((void**)&s->rnbr, (size_t)n * s->rwp * 4));
    V2_CUDA(s->cache->get((void**)&s->vsets, (size_t)2 * s->rwp * 4));
    V2_CUDA(s->cache->get((void**)&s->counters, 4 * sizeof(unsigned long long)));
    int rc = v2_arrays(s, lean, err);
    if (rc == CR_ERR_NOMEM && !lean) rc = v2_arrays(s, true, err);
    if (rc) return rc;
    std::vector<uint32_t> nbr((size_t)n * s->rwp, 0);
    std::vector<uint32_t> rnbr((size_t)n * s->rwp, 0), vsets((size_t)2 * s->rwp, 0);
    for (int v = 0; v < n; ++v) {
        for (uint32_t e = h_rp[v]; e < h_rp[v + 1]; ++e) {
            const int u = h_col[e];
            nbr[(size_t)v * s->rwp + (u >> 5)] |= 1u << (u & 31);
            rnbr[(size_t)u * s->rwp + (v >> 5)] |= 1u << (v & 31);
        }
        const uint32_t deg = h_rp[v + 1] - h_rp[v];
        if (deg <= (uint32_t)k) vsets[v >> 5] |= 1u << (v & 31);
        if (deg == 0) vsets[s->rwp + (v >> 5)] |= 1u << (v & 31);
    }
    V2_CUDA(cudaMemcpyAsync(s->nbr, nbr.data(), nbr.size() * 4, cudaMemcpyHostToDevice, st));
    V2_CUDA(cudaMemcpyAsync(s->rnbr, rnbr.data(), rnbr.size() * 4, cudaMemcpyHostToDevice, st));
    V2_CUDA(cudaMemcpyAsync(s->vsets, vsets.data(), vsets.size() * 4, cudaMemcpyHostToDevice, st));
    return CR_OK;
}

void v2_destroy(V2Solver* s) {
    if (!s) return;
    v2_put_arrays(s);
    void* ptrs[] = {s->table, s->marked, s->nbr, s->val1, s->newval, s->rnbr, s->vsets, s->counters};
    for (void* q : ptrs)
        s->cache->put(q);
    delete s;
}

int v2_init(V2Solver* s, std::string* err) {
    cudaStream_t st = s->st;
    V2_CUDA(cudaEventRecord(s->i0, st));
    V2_CUDA(cudaMemsetAsync(s->table, kUnmarked, (size_t)s->C * s->n, st));
    V2_CUDA(cudaMemsetAsync(s->newval, kV2None, (size_t)s->C * s->n, st));
    V2_CUDA(cudaMemsetAsync(s->val1, kV2None, (size_t)s->C * s->n, st));
    const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((s->C + 255) / 256, (uint64_t)s->num_sms * 4));
    k_v2_init<<<grid, 256, 0, st>>>(s->table, s->marked, s->changed, s->fin1, s->fin2, s->counters, s->configs, s->C, s->n,
                                    s->k, s->rwp);
    V2_CUDA(cudaGetLastError());
    V2_CUDA(cudaEventRecord(s->i1, st));
    s->first = true;
    s->hstats = cr_v2_hash_stats{};
    s->hstats.capacity = s->hcap;
    return CR_OK;
}

// Depth-1 values of the nodes [lo, hi): with a cloud table, fill it and evaluate its nodes
// first.  Returns the kernels launched.
template <int K, int W>
static int launch_v2_val1(V2Solver* s, V2Dev d, uint64_t lo, uint64_t hi, int grid_cfg, size_t sm) {
    cudaStream_t st = s->st;
    raise_smem_limit((const void*)k_v2_val1<K, W>, sm);
    d.node_lo = lo;
    d.node_hi = hi;
    int launches = 0;
    if (d.hkey) {
        raise_smem_limit((const void*)k_v2_hinsert<K, W>, sm);
        raise_smem_limit((const void*)k_v2_heval<K, W>, sm);
        cudaMemsetAsync(d.hkey, 0, d.hcap * sizeof(unsigned long long), st);
        k_v2_hinsert<K, W><<<grid_cfg, 256, sm, st>>>(d);
        const int grid_h = (int)std::max<uint64_t>(1, std::min<uint64_t>((d.hcap + 255) / 256, (uint64_t)s->num_sms * 8));
        k_v2_heval<K, W><<<grid_h, 256, sm, st>>>(d);
        launches += 2;
        ++s->hstats.fills;
    }
    k_v2_val1<K, W><<<grid_cfg, 256, sm, st>>>(d);
    return launches + 1;
}

template <int K, int W>
static int launch_v2_kernels(V2Solver* s, const V2Dev& d, int grid_cfg, size_t sm) {
    int launches = 0;
    if (d.p >= 2 && d.plain) {
        raise_smem_limit((const void*)k_v2_plain<K, W>, sm);
        k_v2_plain<K, W><<<grid_cfg, 256, sm, s->st>>>(d);
        ++launches;
    }
    const uint64_t nodes = (uint64_t)s->C * s->n;
    const uint64_t chunk = d.hkey ? std::max<uint64_t>(1, s->chunk_nodes) : nodes;
    for (uint64_t lo = 0; lo < nodes; lo += chunk)
        launches += launch_v2_val1<K, W>(s, d, lo, std::min(nodes, lo + chunk), grid_cfg, sm);
    if (s->lean) cudaMemsetAsync(s->newval, kV2None, nodes, s->st);   // (it held the unsafe rows)
    raise_smem_limit((const void*)k_v2_root<K, W>, sm);
    k_v2_root<K, W><<<grid_cfg, 256, sm, s->st>>>(d);
    return launches + 1;
}

template <int K>
static int launch_v2_k(V2Solver* s, const V2Dev& d, int W, int grid_cfg, size_t sm) {
    switch (W) {
        case 1: return launch_v2_kernels<K, 1>(s, d, grid_cfg, sm);
        case 2: return launch_v2_kernels<K, 2>(s, d, grid_cfg, sm);
        case 4: return launch_v2_kernels<K, 4>(s, d, grid_cfg, sm);
        case 8: return launch_v2_kernels<K, 8>(s, d, grid_cfg, sm);
        default: return launch_v2_kernels<K, 16>(s, d, grid_cfg, sm);
    }
}

template <int W>
static void launch_v2_begin(const V2Solver* s, const V2Dev& d, int grid, size_t sm) {
    raise_smem_limit((const void*)k_v2_begin<W>, sm);
    k_v2_begin<W><<<grid, 256, sm, s->st>>>(d, s->lev, s->changed);
}

template <int K>
static void launch_dilate(const V2Solver* s, const uint8_t* in, uint8_t* out, int grid) {
    k_v2_dilate<K><<<grid, 256, 0, s->st>>>(in, out, s->configs, s->C, s->n, s->rp, s->col, s->binom);
}

int v2_pass(V2Solver* s, uint64_t* found, cr_solve_stats* stats, std::string* err) {
    cudaStream_t st = s->st;
    V2_CUDA(cudaEventRecord(s->e0, st));
    const V2Dev d = v2_view(s);
    const size_t sm = (size_t)s->n * s->rwp * 4;
    const uint64_t pairs = (uint64_t)s->C * s->n;
    const int grid_cfg = (int)std::max<uint64_t>(1, std::min<uint64_t>((s->C + 7) / 8, (uint64_t)s->num_sms * 8));
    const int grid_cfg_small = (int)std::max<uint64_t>(1, std::min<uint64_t>((s->C + 255) / 256, (uint64_t)s->num_sms * 4));
    int launches = 0;
    if (!s->first) {
        switch (s->W) {
            case 1: launch_v2_begin<1>(s, d, grid_cfg, sm); break;
            case 2: launch_v2_begin<2>(s, d, grid_cfg, sm); break;
            case 4: launch_v2_begin<4>(s, d, grid_cfg, sm); break;
            case 8: launch_v2_begin<8>(s, d, grid_cfg, sm); break;
            default: launch_v2_begin<16>(s, d, grid_cfg, sm); break;
        }
        ++launches;
        for (int j = 1; j < s->p; ++j) {
            const uint8_t* in = s->lev + (size_t)(j - 1) * s->C;
            uint8_t* out = s->lev + (size_t)j * s->C;
            switch (s->k) {
                case 1: launch_dilate<1>(s, in, out, grid_cfg_small); break;
                case 2: launch_dilate<2>(s, in, out, grid_cfg_small); break;
                case 3: launch_dilate<3>(s, in, out, grid_cfg_small); break;
                default: launch_dilate<4>(s, in, out, grid_cfg_small); break;
            }
            ++launches;
        }
    }
    s->first = false;
    switch (s->k) {
        case 1: launches += launch_v2_k<1>(s, d, s->W, grid_cfg, sm); break;
        case 2: launches += launch_v2_k<2>(s, d, s->W, grid_cfg, sm); break;
        case 3: launches += launch_v2_k<3>(s, d, s->W, grid_cfg, sm); break;
        default: launches += launch_v2_k<4>(s, d, s->W, grid_cfg, sm); break;
    }
    if (s->lean) cudaMemsetAsync(s->changed, 0, s->C, st);
    const int grid_apply = (int)std::max<uint64_t>(1, std::min<uint64_t>((pairs + 255) / 256, (uint64_t)s->num_sms * 8));
    k_v2_apply<<<grid_apply, 256, 0, st>>>(s->table, s->marked, s->newval, s->changed, s->C, s->n, s->rwp, s->counters,
                                           s->h_pinned);
    launches += 1;
    V2_CUDA(cudaGetLastError());
    V2_CUDA(cudaEventRecord(s->e1, st));
    V2_CUDA(cudaStreamSynchronize(st));
    *found = s->h_pinned[0];
    s->hstats.child_visits += s->h_pinned[1];
    s->hstats.entries += s->h_pinned[2];
    float ms = 0;
    cudaEventElapsedTime(&ms, s->e0, s->e1);
    stats->main_ms += ms;
    stats->kernel_launches += launches;
    return CR_OK;
}

int v2_load_states(V2Solver* s, const uint8_t* states, std::string* err) {
    cudaStream_t st = s->st;
    V2_CUDA(cudaMemcpyAsync(s->table, states, (size_t)s->C * s->n, cudaMemcpyHostToDevice, st));
    launch_marks_from_table(s->table, s->C, s->n, 1, s->rwp, s->marked, s->num_sms * 8, st);
    V2_CUDA(cudaGetLastError());
    V2_CUDA(cudaStreamSynchronize(st));   // the caller's host buffer goes out of scope
    return CR_OK;
}

void v2_verdict(V2Solver* s, unsigned long long* best_key) {
    const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((s->C + 7) / 8, (uint64_t)s->num_sms * 8));
    launch_verdict_raw(s->table, s->marked, s->C, s->n, s->rw, s->rwp, 1, best_key, grid, s->st);
}

const uint8_t* v2_table(const V2Solver* s) { return s->table; }

cr_v2_hash_stats v2_hash_stats(const V2Solver* s) { return s->hstats; }

}  // namespace crgpu
