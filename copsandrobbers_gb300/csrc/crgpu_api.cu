// crgpu_api.cu - the C ABI of include/crgpu.h: contexts, graph parsing, the v1 solve
// schedule, verdict, table read-out and the table-file writer.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/crgpu.h"
#include "crgpu_internal.cuh"
#include "crgpu_ctx.h"
#include "crgpu_v2.h"

namespace crgpu {
void launch_cop(const V1Dev& d, int col, int nx, int direct, int grid, cudaStream_t st, bool end = false);
void launch_and(const V1Dev& d, int col, bool p1, int grid, cudaStream_t st, const LoopCtl& loop);
void launch_init(const V1Dev& d, bool whole, int grid, cudaStream_t st);
void launch_init_pass1(const V1Dev& d, int num_sms, cudaStream_t st);
void launch_marks_from_table(const uint8_t* table, uint32_t C, int n, int cols, int rwp, uint32_t* marked,
                             int grid, cudaStream_t st);
void launch_game(const uint8_t* table, const uint16_t* configs, const unsigned long long* heads,
                 const unsigned long long* trans, const uint32_t* rp, const uint16_t* adj, int n, int k,
                 long long best, int cap, long long* out_c, int* out_r, int* count, int* captured,
                 cudaStream_t st);
void launch_loop_enter(const V1Dev& d, const LoopCtl& c, int first, int grid, cudaStream_t st);
void launch_verdict(const V1Dev& d, int cols, unsigned long long* best, int grid, cudaStream_t st);
void launch_popcount(const uint32_t* plane, size_t words, unsigned long long* out, int grid,
                     cudaStream_t st);
int max_cop_blocks_per_sm(int k, int rwp, int S);
bool pull_supported(int S, int rwp);
int create_solver(cr_context* ctx, const cr_graph* g, int32_t k, int32_t p, int32_t rules, bool lean, cr_solver** out);
int small_team(const V1Dev& d, double avg_deg);
cudaError_t launch_small_run(const V1Dev& d, const LoopCtl& c, int first, int passes, bool p1, int team, cudaStream_t st);
int cop_launches(int direct);
int cop_launches_k(int direct, bool sep);
size_t cop_smem_bytes(int S, int rwp);
size_t and_smem_bytes(int S, int rwp, int n);
void launch_unrank(const uint32_t* B, int n, int k, uint32_t C, uint16_t* out, int grid, cudaStream_t st);
int trans_cap(int k, int maxdeg);
void launch_trans(int k, const uint16_t* configs, uint32_t C, int n, const uint32_t* rp,
                  const uint16_t* adj, const uint32_t* B, int cap, unsigned long long* counts,
                  const unsigned long long* heads, unsigned long long* data, unsigned int* err,
                  int grid, cudaStream_t st);
void launch_scan(const unsigned long long* in, unsigned long long* out, uint32_t C, cudaStream_t st);
void launch_digest(const uint8_t* table, size_t bytes, unsigned long long* out, int grid, cudaStream_t st);
}  // namespace crgpu

using namespace crgpu;

// A solve's counters on the device, written whole before each initializeCaptures.
struct SolveCtl {
    unsigned long long counters[4];    // [0] pass_new, [1] verdict key, [2] scratch
    unsigned err;
    unsigned sync[kSyncWords];         // V1Dev::sync
    int hist_n;                        // passes recorded since the last k_loop_enter
    unsigned done;                     // V1Dev::done
    int pad[2];
    ColMeta* meta() { return reinterpret_cast<ColMeta*>(this + 1); }
};
// The pass counts go straight to the kit's pinned words, a ring that the host reads as they come;
// the two words behind it take the verdict's and the digest's results.
constexpr int kHistRing = 64;
static_assert(sizeof(SolveCtl) % 16 == 0 && kHistRing + 2 <= cr_solver_kit::kWords, "control block");

// Host images of a solver's small device arrays, laid out one after the other (256-byte aligned)
// and uploaded with one copy.
struct SmallArrays {
    std::vector<uint8_t> bytes;
    std::vector<std::pair<void**, size_t>> at;
    template <typename T, typename D>
    void add(D** slot, const std::vector<T>& v) {
        const size_t off = (bytes.size() + 255) & ~size_t(255);
        bytes.resize(off + std::max<size_t>(v.size() * sizeof(T), 1));
        if (!v.empty()) memcpy(bytes.data() + off, v.data(), v.size() * sizeof(T));
        at.push_back({(void**)slot, off});
    }
    // (the pageable source is staged before the copy call returns)
    cudaError_t upload(cr_block_cache& cache, unsigned char** base, cudaStream_t st) {
        cudaError_t e = cache.get((void**)base, bytes.size());
        if (e == cudaSuccess) e = cudaMemcpyAsync(*base, bytes.data(), bytes.size(), cudaMemcpyHostToDevice, st);
        for (auto& a : at) *a.first = *base + a.second;
        return e;
    }
};

// Per-solve state.  Host copies of the graph are kept for the hop masks and file output.
struct cr_solver {
    cr_context* ctx = nullptr;
    int n = 0, k = 0, p = 0, rules = CR_RULES_V1, cols = 0, rw = 0, rwp = 0, S = 2;
    uint64_t C = 0;
    int maxdeg = 0, mindeg = CR_MAX_N;
    std::vector<uint32_t> h_rp;       // the robber's moves (with self-loops under CR_ROBBER_STAY)
    std::vector<uint16_t> h_col;
    std::vector<uint32_t> h_crp;      // the cops' moves (with self-loops under CR_COP_STAY)
    std::vector<uint16_t> h_ccol;
    bool cop_stay = false, robber_stay = false;
    bool lean = false;                // without what lean_footprint leaves out
    int cop_maxdeg = 0;
    uint32_t forms = CR_FORMS_ALL;    // cr_solver_set_forms
    uint32_t* d_crp = nullptr;        // set only when the two move graphs differ
    uint16_t* d_ccol = nullptr;
    uint32_t* d_ciso = nullptr;
    std::vector<uint32_t> h_binom;
    // device
    uint32_t* d_rp = nullptr;
    uint16_t* d_col = nullptr;
    uint32_t* d_binom = nullptr;
    uint16_t* d_configs = nullptr;
    uint32_t* d_hop = nullptr;
    uint8_t* d_table = nullptr;
    uint32_t* d_marked = nullptr;
    uint32_t* d_front = nullptr;
    uint8_t* d_fflag = nullptr;
    uint32_t* d_cand = nullptr;
    uint32_t* d_h1 = nullptr;   // k = 2, 3, 4: head rows of the separable dense cop turn
    uint32_t* d_cbits = nullptr;      // push-mode candidate bitmap
    uint32_t* d_list = nullptr;       // [cols][C] row lists of the frontiers
    uint32_t* d_clist = nullptr;      // [C] push-mode candidate list
    uint32_t* d_rrp = nullptr;
    uint16_t* d_rcol = nullptr;
    uint32_t* d_nbr = nullptr;
    uint32_t* d_iso = nullptr;
    uint32_t* d_rhop = nullptr;
    uint16_t* d_ell = nullptr;        // hop lists of the last column's tile form
    uint32_t* d_ell_off = nullptr;
    uint32_t* d_cin = nullptr;        // closed in-neighbour words of the first pass's tiles
    uint8_t* d_cover = nullptr;   // first-pass neighbour-slot masks (p = 1, max degree <= 32)
    int cover_w = 0, npad = 0;
    // the small arrays above (graph, rank table, masks) share one block, uploaded at once
    unsigned char* d_small = nullptr;
    // control block: SolveCtl, then the columns' ColMeta
    SolveCtl* d_ctl = nullptr;
    unsigned long long* d_heads = nullptr;
    unsigned long long* d_trans = nullptr;
    uint64_t n_trans = 0;
    cr_solver_kit kit;                // pinned: the ring of pass counts, then two words of results
    bool init_timing = false;         // kit.ev[2], ev[3] bracket an initializeCaptures in flight
    bool unsynced = false;            // the table may still be being written
    bool shared = false;              // the table's address has been given away
    // phase state
    bool initialized = false;
    bool finished = false;
    // p = 1: initializeCaptures is folded into the first pass (one sweep writes the table);
    // set between cr_solver_init and that pass, and undone by materialize_init() when the
    // post-initializeCaptures state is read first
    bool init_pending = false;
    uint64_t base_caps = 0;
    std::vector<uint64_t> pass_counts;
    cr_solve_stats stats{};
    int grid_cop = 1, grid_small = 1;
    crgpu::V2Solver* v2 = nullptr;
};

static int fail(cr_context* ctx, int code, const char* fmt, ...) {
    if (ctx) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(buf, sizeof(buf), fmt, ap);
        va_end(ap);
        ctx->err = buf;
    }
    return code;
}

#define CR_CUDA(ctx, call)                                                                  \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess)                                                              \
            return fail((ctx), CR_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

static uint64_t binom_u64(int64_t n, int64_t k) {
    if (k < 0 || n < 0 || k > n) return 0;
    if (k > n - k) k = n - k;
    unsigned __int128 r = 1;
    for (int64_t i = 1; i <= k; ++i) {
        r = r * (unsigned __int128)(n - i + 1) / (unsigned __int128)i;
        if (r > (unsigned __int128)UINT64_MAX) return UINT64_MAX;
    }
    return (uint64_t)r;
}

extern "C" {

int cr_context_create(int32_t device, void* stream, cr_context** out) {
    if (!out) return CR_ERR_INVALID;
    *out = nullptr;
    cr_context* c = new (std::nothrow) cr_context();
    if (!c) return CR_ERR_NOMEM;
    c->device = device;
    cudaError_t e = cudaSetDevice(device);
    if (e == cudaSuccess) {
        if (stream) {
            c->stream = (cudaStream_t)stream;
        } else {
            e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
            c->own_stream = true;
        }
    }
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess) {
        delete c;
        return CR_ERR_CUDA;
    }
    *out = c;
    return CR_OK;
}

int cr_context_destroy(cr_context* ctx) {
    if (!ctx) return CR_OK;
    if (ctx->own_stream && ctx->stream) cudaStreamDestroy(ctx->stream);
    cudaSetDevice(ctx->device);
    ctx->cache.clear();
    for (cr_solver_kit& k : ctx->kits) k.release();
    delete ctx;
    return CR_OK;
}

const char* cr_context_last_error(const cr_context* ctx) { return ctx ? ctx->err.c_str() : ""; }

int cr_context_set_cache_limit(cr_context* ctx, uint64_t bytes) {
    if (!ctx) return CR_ERR_INVALID;
    CR_CUDA(ctx, cudaSetDevice(ctx->device));
    ctx->cache.set_limit(bytes);
    return CR_OK;
}

// For tests: the device is full once this context's blocks take `bytes`; *peak = the most that solvers
// have taken of them so far.
int cr_context_limit_blocks(cr_context* ctx, uint64_t bytes, uint64_t* peak) {
    if (!ctx) return CR_ERR_INVALID;
    std::lock_guard<std::mutex> lock(ctx->cache.mu);
    ctx->cache.most = bytes;
    if (peak) *peak = ctx->cache.peak_used;
    return CR_OK;
}

int cr_context_set_profiling(cr_context* ctx, int32_t on) {
    if (!ctx) return CR_ERR_INVALID;
    ctx->profiling = on != 0;
    return CR_OK;
}

int cr_graph_parse(const char* text, size_t len, int32_t* n_out, uint32_t* row_ptr,
                   uint16_t* col_idx, size_t col_cap, size_t* nnz_out) {
    // Graph::Graph (lib/src/Graph.cpp:26-70): N = first-line width; '0'/'1' fill row-major;
    // '\n' advances the row only after a digit; '-' ends the matrix; anything else is skipped.
    if (!n_out || !nnz_out || (!text && len)) return CR_ERR_INVALID;
    size_t n = 0;
    while (n < len && text[n] != '\n' && text[n] != '\r' && text[n] != '-') ++n;
    if (n > CR_MAX_N) return CR_ERR_LIMIT;
    *n_out = (int32_t)n;
    std::vector<uint8_t> m(n * n, 0);
    size_t row = 0, col = 0;
    for (size_t i = 0; i < len && n; ++i) {
        char c = text[i];
        if (c == '-') break;
        if (c == '0' || c == '1') {
            if (row < n && col < n) m[row * n + col] = (uint8_t)(c == '1');
            ++col;
        } else if (c == '\n') {
            if (col > 0) { ++row; col = 0; }
        }
    }
    size_t nnz = 0;
    for (uint8_t x : m) nnz += x;
    *nnz_out = nnz;
    if (!row_ptr) return CR_OK;
    if (!col_idx && nnz) return CR_ERR_INVALID;
    if (col_cap < nnz) return CR_ERR_INVALID;
    size_t e = 0;
    row_ptr[0] = 0;
    for (size_t r = 0; r < n; ++r) {
        for (size_t c = 0; c < n; ++c)
            if (m[r * n + c]) col_idx[e++] = (uint16_t)c;
        row_ptr[r + 1] = (uint32_t)e;
    }
    return CR_OK;
}

static int slots_for(int n) { (void)n; return 2; }

// Head rows of the separable dense cop turn (k = 2, 3, 4): every multiset of k - 1 vertices times
// every vertex, one frontier row each; about k/8 of a p = 1 table's bytes.  0 when the turn keeps
// the tuple-gathering form (k = 1, or more than two value slots).
static uint64_t h1_bytes(int n, int k, int S, int rwp) {
    if (k < 2 || S != 2 || !pull_supported(S, rwp)) return 0;
    return binom_u64((int64_t)n + k - 2, k - 1) * n * S * rwp * 4;
}

// The head rows of a solver.  k = 2 and 4 do without them (in the tuple-gathering form) where
// the device or the solver's footprint has no room.
static cudaError_t alloc_h1(cr_solver* s) {
    const uint64_t hb = h1_bytes(s->n, s->k, s->S, s->rwp);
    if (!hb || (s->lean && s->k != 3)) return cudaSuccess;
    const cudaError_t e = s->ctx->cache.get((void**)&s->d_h1, hb);
    return e == cudaErrorMemoryAllocation && s->k != 3 ? cudaSuccess : e;
}

// A block that a solver needs later than its own, in place of what it can do without (head rows of
// k = 2 and 4, the plain values of the v2 rules) where the device has no room for both.
static cudaError_t get_or_shed(cr_solver* s, void** out, size_t bytes) {
    cr_block_cache& cache = s->ctx->cache;
    const cudaError_t e = cache.get(out, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    if (s->v2) {
        if (!crgpu::v2_shed(s->v2)) return e;
    } else {
        if (!s->d_h1 || s->k == 3) return e;
        cache.put(s->d_h1);
        s->d_h1 = nullptr;
    }
    return cache.get(out, bytes);
}

static void layout(int n, int k, int p, int rules, int S, uint64_t* C, int* cols, int* rw, int* rwp) {
    *C = binom_u64((int64_t)n + k - 1, k);
    *cols = rules == CR_RULES_V2 ? 1 : 2 * p;
    *rw = (n + 31) / 32;
    *rwp = round_words(*rw);
    (void)S;
}

uint64_t cr_solver_footprint(int32_t n, int32_t k, int32_t p, int32_t rules) {
    if (n <= 0 || k <= 0 || p <= 0) return 0;
    if (rules == CR_RULES_V2) return crgpu::v2_footprint(n, k, p);
    uint64_t C;
    int cols, rw, rwp;
    const int S = slots_for(n);
    layout(n, k, p, rules, S, &C, &cols, &rw, &rwp);
    uint64_t b = C * (uint64_t)n * cols;                 // table
    b += (uint64_t)cols * C * rwp * 4;                   // marked
    b += (uint64_t)cols * C * S * rwp * 4;               // frontiers
    b += C * S * rwp * 4 + cand_bits_bytes(C) + C * 4;   // push-mode candidate rows, bitmap, list
    b += (uint64_t)cols * C * 4;                         // frontier row lists
    b += h1_bytes(n, k, S, rwp);                         // separable dense cop turn
    b += (uint64_t)cols * C;                             // flags
    b += C * (uint64_t)k * 2;                            // configs
    b += (uint64_t)n * rwp * 4 * 3 + (uint64_t)k * (n + 1) * 4 + (1u << 16);
    b += (uint64_t)n * rw * 64;                          // hop lists of the last column's tiles (at most)
    if (cols == 2) b += 2ull * n * (uint64_t)((n + 7) & ~7) * 4;   // first-pass cover masks
    return b;
}

}  // extern "C"

namespace crgpu {
// Bytes of a lean solve: without the head rows of k = 2 and 4 (the solver then gathers tuples), or the
// plain values of the v2 rules (which are looked up where they are reached).  A server admits by it
// what its budget cannot hold whole.
uint64_t lean_footprint(int n, int k, int p, int rules) {
    if (rules == CR_RULES_V2) return v2_lean_footprint(n, k, p);
    uint64_t C;
    int cols, rw, rwp;
    layout(n, k, p, rules, slots_for(n), &C, &cols, &rw, &rwp);
    return cr_solver_footprint(n, k, p, rules) - (k == 3 ? 0 : h1_bytes(n, k, slots_for(n), rwp));
}
}  // namespace crgpu

extern "C" {

static void free_v1(cr_solver* s) {
    void* ptrs[] = {s->d_small, s->d_ctl, s->d_configs, s->d_table, s->d_marked, s->d_front, s->d_fflag, s->d_heads,
                    s->d_trans, s->d_cand, s->d_cbits, s->d_list, s->d_clist, s->d_h1};
    for (void* q : ptrs) s->ctx->cache.put(q);   // the context keeps them for the next solver
    s->ctx->put_kit(s->kit);
}

static V1Dev dev_view(const cr_solver* s) {
    V1Dev d;
    d.g.n = s->n;
    d.g.rw = s->rw;
    d.g.rwp = s->rwp;
    d.g.row_ptr = s->d_rp;
    d.g.col = s->d_col;
    d.g.rrow_ptr = s->d_rrp;
    d.g.rcol = s->d_rcol;
    d.g.nbr = s->d_nbr;
    d.g.isolated = s->d_iso;
    d.g.rhop = s->d_rhop;
    d.g.ell = s->d_ell;
    d.g.ell_off = s->d_ell_off;
    d.g.cin = s->d_cin;
    d.g.maxdeg = s->maxdeg;
    d.g.mindeg = s->mindeg;
    d.g.cover = s->d_cover;
    d.g.cover_w = s->cover_w;
    d.g.npad = s->npad;
    d.g.nnz = (int)s->h_col.size();
    d.g.cop_row_ptr = s->d_crp;
    d.g.cop_col = s->d_ccol;
    d.g.cop_isolated = s->d_ciso;
    d.k = s->k;
    d.cols = s->cols;
    d.S = s->S;
    d.C = (uint32_t)s->C;
    d.binom = s->d_binom;
    d.configs = s->d_configs;
    d.hop = s->d_hop;
    d.table = s->d_table;
    d.marked = s->d_marked;
    d.front = s->d_front;
    d.fflag = s->d_fflag;
    d.cand = s->d_cand;
    d.h1 = s->d_h1;
    d.cbits = s->d_cbits;
    // forms switched off: no head rows (the tuple pull), a push ratio that always or never
    // pushes, the last column's general form
    if (!(s->forms & CR_FORM_SEPARABLE)) d.h1 = nullptr;
    if (d.h1) d.push_ratio = kPushRatioSeparable;
    if (!(s->forms & CR_FORM_PULL)) d.push_ratio = 0u;
    else if (!(s->forms & CR_FORM_PUSH)) d.push_ratio = 0xFFFFFFFFu;
    d.fresh_last = (s->forms & CR_FORM_FRESH_LAST) ? 1 : 0;
    d.list = s->d_list;
    d.clist = s->d_clist;
    d.sync = s->d_ctl->sync;      // (addresses only)
    d.meta = s->d_ctl->meta();
    d.pass_new = s->d_ctl->counters;
    d.err = &s->d_ctl->err;
    d.done = &s->d_ctl->done;
    return d;
}

// Exact-p-hop vertex sets (k_cops_visibility.cpp:245-262, robber self-edges off).
static std::vector<uint32_t> hop_masks(const cr_solver* s) {
    std::vector<uint32_t> hop((size_t)s->n * s->rwp, 0);
    std::vector<uint8_t> cur(s->n), nxt(s->n);
    for (int r = 0; r < s->n; ++r) {
        std::fill(cur.begin(), cur.end(), 0);
        cur[r] = 1;
        for (int step = 0; step < s->p; ++step) {
            std::fill(nxt.begin(), nxt.end(), 0);
            for (int v = 0; v < s->n; ++v)
                if (cur[v])
                    for (uint32_t e = s->h_rp[v]; e < s->h_rp[v + 1]; ++e) nxt[s->h_col[e]] = 1;
            cur.swap(nxt);
        }
        for (int v = 0; v < s->n; ++v)
            if (cur[v]) hop[(size_t)r * s->rwp + (v >> 5)] |= 1u << (v & 31);
    }
    return hop;
}

static int alloc_v1(cr_solver* s, SmallArrays& small) {
    cr_context* ctx = s->ctx;
    const size_t C = s->C;
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_table, C * s->n * s->cols));
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_marked, (size_t)s->cols * C * s->rwp * 4));
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_front, (size_t)s->cols * C * s->S * s->rwp * 4));
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_fflag, (size_t)s->cols * C));
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_cand, C * s->S * s->rwp * 4));
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_cbits, cand_bits_bytes(C)));
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_list, (size_t)s->cols * C * 4));
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_clist, C * 4));
    CR_CUDA(ctx, cudaMemsetAsync(s->d_cand, 0, C * s->S * s->rwp * 4, ctx->stream));
    CR_CUDA(ctx, cudaMemsetAsync(s->d_cbits, 0, cand_bits_bytes(C), ctx->stream));
    std::vector<uint32_t> hop = hop_masks(s);
    small.add(&s->d_hop, hop);
    // transposed hop masks (bit r of row u iff u in hop(r)), and hop(r) as lists
    std::vector<uint32_t> rhop(hop.size(), 0), list_at(s->n + 1, 0);
    std::vector<uint16_t> lists;
    for (int r = 0; r < s->n; ++r) {
        for (int w = 0; w < s->rw; ++w)
            for (uint32_t b = hop[(size_t)r * s->rwp + w]; b; b &= b - 1) {
                const int u = w * 32 + __builtin_ctz(b);
                rhop[(size_t)u * s->rwp + (r >> 5)] |= 1u << (r & 31);
                lists.push_back((uint16_t)u);
            }
        list_at[r + 1] = (uint32_t)lists.size();
    }
    small.add(&s->d_rhop, rhop);
    // the lists padded and 32 vertices side by side (the last column's tile form)
    std::vector<uint32_t> ell_off(s->rw + 1, 0);
    for (int w = 0; w < s->rw; ++w) {
        uint32_t longest = 0;
        for (int r = w * 32; r < std::min(w * 32 + 32, s->n); ++r) longest = std::max(longest, list_at[r + 1] - list_at[r]);
        ell_off[w + 1] = ell_off[w] + longest;
    }
    std::vector<uint16_t> ell((size_t)ell_off[s->rw] * 32, (uint16_t)(s->rw * 32));
    for (int r = 0; r < s->n; ++r)
        for (uint32_t e = list_at[r]; e < list_at[r + 1]; ++e)
            ell[(size_t)(ell_off[r >> 5] + e - list_at[r]) * 32 + (r & 31)] = lists[e];
    small.add(&s->d_ell, ell);
    small.add(&s->d_ell_off, ell_off);
    // the cops' out-neighbour masks (capture-seed closed form) and their in-neighbour CSR
    // (push mode), both of the cops' move graph
    const std::vector<uint32_t>& crp = s->h_crp;
    const std::vector<uint16_t>& ccol = s->h_ccol;
    std::vector<uint32_t> nbr((size_t)s->n * s->rwp, 0);
    std::vector<uint32_t> rrp(s->n + 1, 0);
    for (uint32_t e = 0; e < ccol.size(); ++e) rrp[ccol[e] + 1]++;
    for (int v = 0; v < s->n; ++v) rrp[v + 1] += rrp[v];
    std::vector<uint16_t> rcol(std::max<size_t>(ccol.size(), 1));
    std::vector<uint32_t> fill(rrp.begin(), rrp.end() - 1);
    for (int u = 0; u < s->n; ++u)
        for (uint32_t e = crp[u]; e < crp[u + 1]; ++e) {
            const int v = ccol[e];
            nbr[(size_t)u * s->rwp + (v >> 5)] |= 1u << (v & 31);
            rcol[fill[v]++] = (uint16_t)u;  // in-neighbours of v, ascending u
        }
    // robbers without a walk of p moves (the last column's vacuous AND), cops without a move
    std::vector<uint32_t> iso(s->rwp, 0), ciso(s->rwp, 0);
    for (int v = 0; v < s->n; ++v) {
        if (list_at[v + 1] == list_at[v]) iso[v >> 5] |= 1u << (v & 31);
        if (crp[v + 1] == crp[v]) ciso[v >> 5] |= 1u << (v & 31);
    }
    if (s->cop_stay != s->robber_stay) {
        small.add(&s->d_crp, crp);
        small.add(&s->d_ccol, ccol);
        small.add(&s->d_ciso, ciso);
    }
    bool all_move = true;
    for (uint32_t w : ciso) all_move &= w == 0;
    if (s->cols == 2 && s->n >= 16 && all_move) {
        std::vector<uint32_t> cin((size_t)s->rw * s->rw * 32, 0);
        for (int c = 0; c < s->n; ++c) {
            uint32_t* row = cin.data() + (size_t)(c >> 5) * s->rw * 32;
            const uint32_t bit = 1u << (c & 31);
            row[c] |= bit;
            for (uint32_t e = crp[c]; e < crp[c + 1]; ++e) row[ccol[e]] |= bit;
        }
        small.add(&s->d_cin, cin);
    }
    small.add(&s->d_iso, iso);
    small.add(&s->d_nbr, nbr);
    small.add(&s->d_rrp, rrp);
    small.add(&s->d_rcol, rcol);
    // uncovered-slot masks of the folded first pass (two columns, out-degrees <= 32), bit j
    // for the j-th out-neighbour of r: plane 0 [c][r] slots of r outside {c} + N(c), plane 1
    // [c][r] slots of r other than c; masks of cover_w bytes, rows padded to npad robbers
    s->cover_w = 0;
    if (s->cols == 2 && s->maxdeg <= 32) {
        const int W = s->maxdeg <= 8 ? 1 : (s->maxdeg <= 16 ? 2 : 4);
        const int n = s->n, npad = (n + 7) & ~7;
        const size_t plane = (size_t)n * npad;
        std::vector<uint32_t> m(2 * plane, 0);
        for (int r = 0; r < n; ++r) {
            const uint32_t e0 = s->h_rp[r], deg = s->h_rp[r + 1] - e0;
            const uint32_t all = deg == 32 ? 0xFFFFFFFFu : ((1u << deg) - 1u);
            for (int c = 0; c < n; ++c) m[(size_t)c * npad + r] = m[plane + (size_t)c * npad + r] = all;
            for (uint32_t j = 0; j < deg; ++j) {
                const int v = s->h_col[e0 + j];
                m[plane + (size_t)v * npad + r] &= ~(1u << j);   // slot j of r is the cop v
                m[(size_t)v * npad + r] &= ~(1u << j);           // ... and so lies in N[v]
                // slot j of r lies in N(c) for every c with v in N(c), i.e. c an in-neighbour of v
                for (uint32_t f = rrp[v]; f < rrp[v + 1]; ++f) m[(size_t)rcol[f] * npad + r] &= ~(1u << j);
            }
        }
        // plane 0 as the first pass's fast test wants it: a cop's own entry [c][c] all ones (a
        // robber on a cop is never a column-1 mark, so the entry's value is otherwise unused)
        // and the rows of cops that cannot move zero (those rows are read only when every cop
        // of the configuration can move)
        const uint32_t ones = W == 4 ? 0xFFFFFFFFu : ((1u << (8 * W)) - 1u);
        for (int c = 0; c < n; ++c) {
            m[(size_t)c * npad + c] = ones;
            if (crp[c + 1] == crp[c])
                for (int r = 0; r < npad; ++r) m[(size_t)c * npad + r] = 0u;
        }
        std::vector<uint8_t> bytes(m.size() * W);
        for (size_t i = 0; i < m.size(); ++i)
            for (int b = 0; b < W; ++b) bytes[i * W + b] = (uint8_t)(m[i] >> (8 * b));
        small.add(&s->d_cover, bytes);
        s->cover_w = W;
        s->npad = npad;
    }
    return CR_OK;
}

}  // extern "C"

// A solver for (g, k, p, rules); lean = one that holds lean_footprint bytes.
int crgpu::create_solver(cr_context* ctx, const cr_graph* g, int32_t k, int32_t p, int32_t rules, bool lean,
                         cr_solver** out) {
    if (!ctx || !g || !out) return CR_ERR_INVALID;
    *out = nullptr;
    if (g->n <= 0) return fail(ctx, CR_ERR_INVALID, "Graph is empty or failed to load.");
    if (g->n > CR_MAX_N) return fail(ctx, CR_ERR_LIMIT, "n=%d exceeds %d vertices", g->n, CR_MAX_N);
    if (k <= 0 || k > CR_MAX_K) return fail(ctx, CR_ERR_LIMIT, "k=%d outside 1..%d", k, CR_MAX_K);
    if (p <= 0 || p > 63) return fail(ctx, CR_ERR_INVALID, "p=%d outside 1..63", p);
    const int stay = rules & (CR_COP_STAY | CR_ROBBER_STAY);
    const int base_rules = rules & ~(CR_COP_STAY | CR_ROBBER_STAY);
    if (base_rules != CR_RULES_V1 && base_rules != CR_RULES_V2) return fail(ctx, CR_ERR_INVALID, "unknown rules %d", rules);
    if (stay && base_rules != CR_RULES_V1) return fail(ctx, CR_ERR_LIMIT, "stay-allowed rules need CR_RULES_V1");
    if (!g->row_ptr || (g->row_ptr[g->n] && !g->col_idx)) return fail(ctx, CR_ERR_INVALID, "graph arrays missing");
    for (int v = 0; v < g->n; ++v)
        if (g->row_ptr[v + 1] < g->row_ptr[v]) return fail(ctx, CR_ERR_INVALID, "row_ptr not monotone");
    for (uint32_t e = 0; e < g->row_ptr[g->n]; ++e)
        if (g->col_idx[e] >= g->n) return fail(ctx, CR_ERR_INVALID, "neighbour index out of range");
    CR_CUDA(ctx, cudaSetDevice(ctx->device));

    cr_solver* s = new (std::nothrow) cr_solver();
    if (!s) return fail(ctx, CR_ERR_NOMEM, "host allocation failed");
    s->ctx = ctx;
    s->n = g->n;
    s->k = k;
    s->p = p;
    s->rules = base_rules;
    rules = base_rules;
    s->lean = lean;
    s->cop_stay = (stay & CR_COP_STAY) != 0;
    s->robber_stay = (stay & CR_ROBBER_STAY) != 0;
    s->S = slots_for(g->n);
    layout(s->n, k, p, rules, s->S, &s->C, &s->cols, &s->rw, &s->rwp);
    if (s->C == 0 || s->C >= (1ull << 32)) {
        delete s;
        return fail(ctx, CR_ERR_LIMIT, "config count C(%d,%d) outside 1..2^32-1", g->n + k - 1, k);
    }
    // the two move graphs: the input graph, plus a self-loop per vertex for a side that may stay
    auto move_graph = [&](bool self, std::vector<uint32_t>& rp, std::vector<uint16_t>& col) {
        rp.assign(1, 0);
        col.clear();
        for (int v = 0; v < g->n; ++v) {
            bool placed = !self;
            for (uint32_t e = g->row_ptr[v]; e < g->row_ptr[v + 1]; ++e) {
                if (!placed && g->col_idx[e] >= v) {
                    col.push_back((uint16_t)v);
                    placed = true;
                }
                col.push_back(g->col_idx[e]);
            }
            if (!placed) col.push_back((uint16_t)v);
            rp.push_back((uint32_t)col.size());
        }
    };
    move_graph(s->robber_stay, s->h_rp, s->h_col);
    move_graph(s->cop_stay, s->h_crp, s->h_ccol);
    for (int v = 0; v < s->n; ++v) {
        s->maxdeg = std::max<int>(s->maxdeg, s->h_rp[v + 1] - s->h_rp[v]);
        s->mindeg = std::min<int>(s->mindeg, s->h_rp[v + 1] - s->h_rp[v]);
        s->cop_maxdeg = std::max<int>(s->cop_maxdeg, s->h_crp[v + 1] - s->h_crp[v]);
    }
    // B[i][x] = C(n - x + k - 1 - i, k - i)
    s->h_binom.assign((size_t)k * (s->n + 1), 0);
    for (int i = 0; i < k; ++i)
        for (int x = 0; x <= s->n; ++x)
            s->h_binom[(size_t)i * (s->n + 1) + x] = (uint32_t)binom_u64((int64_t)s->n - x + k - 1 - i, k - i);

    auto bail = [&](int code) {
        free_v1(s);
        if (s->v2) crgpu::v2_destroy(s->v2);
        delete s;
        return code;
    };
#define CR_TRY(call)                                                                         \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess) {                                                             \
            fail(ctx, e_ == cudaErrorMemoryAllocation ? CR_ERR_NOMEM : CR_ERR_CUDA, "%s: %s", \
                 #call, cudaGetErrorString(e_));                                             \
            return bail(e_ == cudaErrorMemoryAllocation ? CR_ERR_NOMEM : CR_ERR_CUDA);       \
        }                                                                                    \
    } while (0)
    SmallArrays small;
    small.add(&s->d_rp, s->h_rp);
    small.add(&s->d_col, s->h_col);
    small.add(&s->d_binom, s->h_binom);
    CR_TRY(ctx->get_kit(&s->kit));
    CR_TRY(ctx->cache.get((void**)&s->d_configs, s->C * k * 2));
    CR_TRY(ctx->cache.get((void**)&s->d_ctl, sizeof(SolveCtl) + sizeof(ColMeta) * s->cols));
    CR_TRY(cudaMemsetAsync(s->d_ctl, 0, sizeof(SolveCtl), ctx->stream));
    if (rules == CR_RULES_V1) {
        if (!pull_supported(s->S, s->rwp))
            return (fail(ctx, CR_ERR_LIMIT, "v1 rules: rows of %d vertices exceed the warp layout (n <= 512)", s->n), bail(CR_ERR_LIMIT));
        int rc = alloc_v1(s, small);
        if (rc) return bail(rc);
        CR_TRY(small.upload(ctx->cache, &s->d_small, ctx->stream));
        CR_TRY(alloc_h1(s));   // (last: the rest has to fit without it)
        const int per_sm = max_cop_blocks_per_sm(k, s->rwp, s->S);
        s->grid_cop = (int)std::max<uint64_t>(1, std::min<uint64_t>((s->C + 7) / 8, (uint64_t)ctx->num_sms * per_sm));
        s->grid_small = (int)std::max<uint64_t>(1, std::min<uint64_t>((s->C + 255) / 256, (uint64_t)ctx->num_sms * 4));
        if (and_smem_bytes(s->S, s->rwp, s->n) > 48 * 1024 || cop_smem_bytes(s->S, s->rwp) > 48 * 1024)
            return (fail(ctx, CR_ERR_LIMIT, "shared memory layout too large"), bail(CR_ERR_LIMIT));
    } else {
        CR_TRY(small.upload(ctx->cache, &s->d_small, ctx->stream));
        int rc = crgpu::v2_create(&s->v2, &ctx->cache, s->kit, ctx->stream, ctx->num_sms, s->n, k, p, s->d_rp, s->d_col,
                                  s->h_rp.data(), s->h_col.data(), s->d_binom, s->d_configs,
                                  (uint32_t)s->C, lean, &ctx->err);
        if (rc) return bail(rc);
    }
    const int grid = (int)std::min<uint64_t>((s->C + 255) / 256, (uint64_t)ctx->num_sms * 8);
    launch_unrank(s->d_binom, s->n, k, (uint32_t)s->C, s->d_configs, std::max(grid, 1), ctx->stream);
    CR_TRY(cudaGetLastError());
#undef CR_TRY
    s->stats.slots = s->S;
    *out = s;
    return CR_OK;
}

extern "C" {

int cr_solver_create(cr_context* ctx, const cr_graph* g, int32_t k, int32_t p, int32_t rules,
                     cr_solver** out) {
    return crgpu::create_solver(ctx, g, k, p, rules, false, out);
}

int cr_solver_destroy(cr_solver* s) {
    if (!s) return CR_OK;
    cudaSetDevice(s->ctx->device);
    free_v1(s);
    if (s->v2) crgpu::v2_destroy(s->v2);
    delete s;
    return CR_OK;
}

static int check_err(cr_solver* s, unsigned* bits) {
    cr_context* ctx = s->ctx;
    unsigned e = 0;
    CR_CUDA(ctx, cudaMemcpyAsync(&e, &s->d_ctl->err, sizeof(e), cudaMemcpyDeviceToHost, ctx->stream));
    CR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    *bits = e;
    return CR_OK;
}

// The control block of a fresh solve: zeros and the columns' states.
static int reset_ctl(cr_solver* s, const std::vector<ColMeta>& meta) {
    cr_context* ctx = s->ctx;
    std::vector<unsigned char> h(sizeof(SolveCtl) + sizeof(ColMeta) * meta.size(), 0);
    memcpy(h.data() + sizeof(SolveCtl), meta.data(), sizeof(ColMeta) * meta.size());
    CR_CUDA(ctx, cudaMemcpyAsync(s->d_ctl, h.data(), h.size(), cudaMemcpyHostToDevice, ctx->stream));
    return CR_OK;
}

// Takes up the time of an initializeCaptures whose events have been recorded (they have completed,
// or are waited for).
static void settle_init_time(cr_solver* s) {
    if (!s->init_timing) return;
    s->init_timing = false;
    float ms = 0;
    if (cudaEventSynchronize(s->kit.ev[3]) == cudaSuccess) cudaEventElapsedTime(&ms, s->kit.ev[2], s->kit.ev[3]);
    s->stats.init_ms = ms;
}

// Every configuration contributes its distinct cop vertices, and n * (multisets containing a given
// vertex) = n * (C(n+k-1, k) - C(n+k-2, k)).
static uint64_t base_capture_count(const cr_solver* s) {
    return (uint64_t)s->n * (binom_u64(s->n + s->k - 1, s->k) - binom_u64(s->n + s->k - 2, s->k));
}

// v1 initializeCaptures on the device (enqueued).
static int v1_init(cr_solver* s) {
    cr_context* ctx = s->ctx;
    cudaStream_t st = ctx->stream;
    const size_t C = s->C;
    settle_init_time(s);
    CR_CUDA(ctx, cudaEventRecord(s->kit.ev[2], st));
    CR_CUDA(ctx, cudaMemsetAsync(s->d_table, kUnmarked, C * s->n * s->cols, st));
    V1Dev d = dev_view(s);
    launch_init(d, true, s->grid_small, st);
    CR_CUDA(ctx, cudaGetLastError());
    CR_CUDA(ctx, cudaEventRecord(s->kit.ev[3], st));
    s->init_timing = true;
    s->unsynced = true;
    s->stats.kernel_launches = 1;
    return CR_OK;
}

// initializeCaptures and pass 1 of a p = 1 solve in one kernel (init_pass1_single /
// init_pass1_body): every table byte, both marked planes and both flag planes are written whole
// (column 1's frontier rows where they gained marks), so nothing is cleared first.
static int v1_init_pass1(cr_solver* s) {
    cr_context* ctx = s->ctx;
    cudaStream_t st = ctx->stream;
    settle_init_time(s);
    // column 0's frontier after pass 1 is every row (the implicit list), already consumed by
    // the fused last column, which leaves its flags clear; column 1's list is built from its
    // flags after the kernel (k_loop_enter)
    const std::vector<ColMeta> meta = {ColMeta{0, 0, 0, 0, (int)std::min<uint64_t>(s->C, INT32_MAX), 0, -1, 1},
                                       ColMeta{1, kEmptyLo, -1, 0, 0, 0, 0, 0, 0, 1}};
    if (int rc = reset_ctl(s, meta)) return rc;
    V1Dev d = dev_view(s);
    CR_CUDA(ctx, cudaEventRecord(s->kit.ev[2], st));
    launch_init_pass1(d, ctx->num_sms, st);
    CR_CUDA(ctx, cudaGetLastError());
    CR_CUDA(ctx, cudaEventRecord(s->kit.ev[3], st));
    s->init_timing = true;
    s->init_pending = false;
    s->unsynced = true;
    s->stats.kernel_launches += 1;
    return CR_OK;
}

// The exact post-initializeCaptures state, for a caller that reads the table before pass 1.
static int materialize_init(cr_solver* s) {
    if (!s->init_pending) return CR_OK;
    if (int rc = v1_init(s)) return rc;
    s->init_pending = false;
    return CR_OK;
}

// Enqueue one pass.  Each column's prep rides on the launches of the column before it (column 0's
// ran in k_loop_enter or in the previous pass's last column, which also records the pass's count):
// three launches per cop turn and robber turn.  Profiling: each cop turn is timed with events.
static int v1_enqueue_pass(cr_solver* s, const LoopCtl& loop) {
    cr_context* ctx = s->ctx;
    cudaStream_t st = ctx->stream;
    V1Dev d = dev_view(s);
    for (int col = 0; col < s->cols; ++col) {
        const int nx = (col + 1) % s->cols;
        if (col % 2 == 0) {
            if (ctx->profiling) {
                settle_init_time(s);
                CR_CUDA(ctx, cudaEventRecord(s->kit.ev[2], st));
            }
            launch_cop(d, col, nx, 0, s->grid_cop, st, true);
            if (ctx->profiling) CR_CUDA(ctx, cudaEventRecord(s->kit.ev[3], st));
        } else if (col < s->cols - 1) {
            launch_cop(d, col, nx, 1, s->grid_cop, st, true);
        } else {
            launch_and(d, col, s->p == 1, s->grid_cop, st, loop);
        }
        CR_CUDA(ctx, cudaGetLastError());
        if (ctx->profiling && col % 2 == 0) {
            CR_CUDA(ctx, cudaEventSynchronize(s->kit.ev[3]));
            float ms = 0;
            cudaEventElapsedTime(&ms, s->kit.ev[2], s->kit.ev[3]);
            s->stats.cop_step_ms += ms;
            s->stats.cop_step_launches += 1;
        }
    }
    return CR_OK;
}

// Waits until a pass has written its word of the ring: the word changes, or the stream runs empty
// or fails without that.
static int await_count(cr_solver* s, int slot, unsigned long long* value) {
    cr_context* ctx = s->ctx;
    volatile unsigned long long* word = s->kit.pinned + slot;
    for (unsigned spin = 1; *word == kHistEmpty; ++spin) {
        if (spin % 1024) continue;
        std::this_thread::yield();
        const cudaError_t e = cudaStreamQuery(ctx->stream);
        if (e != cudaErrorNotReady && *word == kHistEmpty)
            return fail(ctx, CR_ERR_CUDA, "a pass recorded nothing: %s", cudaGetErrorString(e));
    }
    *value = *word;
    return CR_OK;
}

static int grow_slots_and_replay(cr_solver* s);

constexpr unsigned long long kFewMarks = 1u << 15;   // the passes of the sparse ends of the solves measured

// Up to `passes` passes, the fused first pass among them when it is pending, until one finds
// nothing.  The host enqueues `ahead` passes beyond the one whose count it waits for, so that the
// device does not idle while the count travels (about 10 us to the host and back); passes behind
// the fixed point return at once, but cost their 3p launches.  So it goes ahead by one pass at
// first, then by `ahead`, and no more once a pass finds little: the end is then near.  Appends the counts to pass_counts, sets finished; widens the value slots and
// replays when a pass overflowed them (that pass is not counted).
static int v1_advance(cr_solver* s, size_t passes, size_t ahead) {
    cr_context* ctx = s->ctx;
    cudaStream_t st = ctx->stream;
    CR_CUDA(ctx, cudaEventRecord(s->kit.ev[0], st));
    const bool first = s->init_pending;
    const int team = ctx->profiling ? 0 : small_team(dev_view(s), (double)s->h_ccol.size() / s->n);
    if (team) passes = std::min<size_t>(passes, kHistRing);
    for (size_t i = 0; i < (team ? passes : 1); ++i) s->kit.pinned[i] = kHistEmpty;
    if (first) {
        if (int rc = v1_init_pass1(s)) return rc;
    }
    const LoopCtl loop{s->kit.pinned, &s->d_ctl->hist_n, kHistRing};
    size_t sent = first ? 1 : 0, got = 0, lead = ahead ? 1 : 0;
    unsigned long long f = 0;
    if (team) {   // all of them in one launch
        CR_CUDA(ctx, launch_small_run(dev_view(s), loop, first ? 1 : 0, (int)passes, s->p == 1, team, st));
        CR_CUDA(ctx, cudaStreamSynchronize(st));
        for (; got < passes && !s->finished; ++got) {
            f = s->kit.pinned[got];
            if (f == kHistEmpty) return fail(ctx, CR_ERR_INTERNAL, "a pass recorded nothing");
            if (f & kHistError) break;
            s->pass_counts.push_back(f);
            s->finished = f == 0;
        }
    } else {
        launch_loop_enter(dev_view(s), loop, first ? 1 : 0, s->grid_small, st);
        CR_CUDA(ctx, cudaGetLastError());
    }
    while (!team && got < passes && !s->finished) {
        for (; sent < passes && sent < got + 1 + lead; ++sent) {
            s->kit.pinned[sent % kHistRing] = kHistEmpty;
            if (int rc = v1_enqueue_pass(s, loop)) return rc;
        }
        if (int rc = await_count(s, (int)(got % kHistRing), &f)) return rc;
        if (f & kHistError) break;
        ++got;
        s->pass_counts.push_back(f);
        s->finished = f == 0;
        lead = f < kFewMarks ? 0 : ahead;
    }
    CR_CUDA(ctx, cudaEventRecord(s->kit.ev[1], st));
    CR_CUDA(ctx, cudaStreamSynchronize(st));   // (the passes sent ahead; the ring is free again)
    s->unsynced = false;
    float ms = 0;
    cudaEventElapsedTime(&ms, s->kit.ev[0], s->kit.ev[1]);
    s->stats.main_ms += ms;
    settle_init_time(s);
    int per_pass = 0;
    for (int col = 0; col < s->cols; ++col)
        per_pass += col % 2 == 0 ? cop_launches_k(0, s->d_h1 != nullptr && (s->forms & CR_FORM_SEPARABLE)) : (col < s->cols - 1 ? cop_launches(1) : 1);
    // (and k_loop_enter, or the small solve's one launch)
    s->stats.kernel_launches += (int64_t)per_pass * (int64_t)(sent - (first ? 1 : 0)) + 1;
    s->stats.passes = (int)s->pass_counts.size();
    if (f & kHistError) {
        if (f & kErrRank) return fail(ctx, CR_ERR_INTERNAL, "successor rank out of range");
        if (f & kErrSlot) return grow_slots_and_replay(s);
        return fail(ctx, CR_ERR_INTERNAL, "device error bits 0x%x", (unsigned)f);
    }
    return CR_OK;
}

// A caller that holds the table's address may read it from another stream.
static int wait_for_table(cr_solver* s) {
    if (!s->unsynced) return CR_OK;
    CR_CUDA(s->ctx, cudaStreamSynchronize(s->ctx->stream));
    s->unsynced = false;
    return CR_OK;
}

int cr_solver_init(cr_solver* s, uint64_t* base_captures) {
    if (!s) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    CR_CUDA(ctx, cudaSetDevice(ctx->device));
    uint64_t caps = 0;
    s->init_pending = false;
    int rc = CR_OK;
    if (s->rules == CR_RULES_V1 && s->cols == 2 && s->S >= 2 && s->cover_w > 0 && (s->forms & CR_FORM_FUSED_FIRST)) {
        // folded into pass 1
        caps = base_capture_count(s);
        s->init_pending = true;
        s->init_timing = false;
        s->stats.init_ms = 0;
        s->stats.kernel_launches = 0;
    } else {
        caps = base_capture_count(s);
        if (s->rules == CR_RULES_V1) {
            rc = v1_init(s);
        } else {
            settle_init_time(s);
            rc = crgpu::v2_init(s->v2, &ctx->err);
            s->init_timing = s->unsynced = !rc;
            s->stats.kernel_launches = 1;
        }
        if (!rc && s->shared) rc = wait_for_table(s);
    }
    if (rc) return rc;
    s->base_caps = caps;
    s->pass_counts.clear();
    s->initialized = true;
    s->finished = false;
    s->stats.main_ms = 0;
    s->stats.cop_step_ms = 0;
    s->stats.cop_step_launches = 0;
    s->stats.passes = 0;
    if (base_captures) *base_captures = caps;
    return CR_OK;
}

static int grow_slots_and_replay(cr_solver* s) {
    // A frontier needed more value slots than allocated: widen and replay from the start.
    cr_context* ctx = s->ctx;
    if (s->S >= 8) return fail(ctx, CR_ERR_INTERNAL, "frontier value range exceeds 8 slots");
    const std::vector<uint64_t> done = s->pass_counts;
    ctx->cache.put(s->d_front);
    s->d_front = nullptr;
    ctx->cache.put(s->d_cand);
    s->d_cand = nullptr;
    ctx->cache.put(s->d_h1);
    s->d_h1 = nullptr;
    s->S *= 2;
    if (!pull_supported(s->S, s->rwp))
        return fail(ctx, CR_ERR_LIMIT, "row too wide for %d value slots", s->S);
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_front, (size_t)s->cols * s->C * s->S * s->rwp * 4));
    CR_CUDA(ctx, ctx->cache.get((void**)&s->d_cand, (size_t)s->C * s->S * s->rwp * 4));
    CR_CUDA(ctx, cudaMemsetAsync(s->d_cand, 0, (size_t)s->C * s->S * s->rwp * 4, ctx->stream));
    CR_CUDA(ctx, cudaMemsetAsync(s->d_cbits, 0, cand_bits_bytes(s->C), ctx->stream));
    CR_CUDA(ctx, alloc_h1(s));
    const int per_sm = max_cop_blocks_per_sm(s->k, s->rwp, s->S);
    s->grid_cop = (int)std::max<uint64_t>(1, std::min<uint64_t>((s->C + 7) / 8, (uint64_t)ctx->num_sms * per_sm));
    if (int rc = v1_init(s)) return rc;
    s->stats.slots = s->S;
    s->pass_counts.clear();
    while (s->pass_counts.size() < done.size()) {
        if (int rc = v1_advance(s, done.size() - s->pass_counts.size(), 2)) return rc;
        if (s->finished) break;
    }
    if (s->pass_counts != done) return fail(ctx, CR_ERR_INTERNAL, "replay diverged within %zu passes", done.size());
    return CR_OK;
}

int cr_solver_pass(cr_solver* s, uint64_t* new_wins) {
    if (!s || !new_wins) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    if (!s->initialized) return fail(ctx, CR_ERR_STATE, "initializeCaptures has not run");
    if (s->finished) { *new_wins = 0; return CR_OK; }
    CR_CUDA(ctx, cudaSetDevice(ctx->device));
    uint64_t f = 0;
    if (s->rules == CR_RULES_V2) {
        int rc = crgpu::v2_pass(s->v2, &f, &s->stats, &ctx->err);
        if (rc) return rc;
        s->unsynced = false;
        settle_init_time(s);
    } else {
        // (a pass that overflows its value slots is not counted: the slots are widened, and it runs
        // again)
        const size_t before = s->pass_counts.size();
        for (int attempt = 0; s->pass_counts.size() == before; ++attempt) {
            if (attempt > 4) return fail(ctx, CR_ERR_INTERNAL, "value slots kept overflowing");
            if (int rc = v1_advance(s, 1, 0)) return rc;
        }
        *new_wins = s->pass_counts.back();
        return CR_OK;
    }
    s->pass_counts.push_back(f);
    s->stats.passes = (int)s->pass_counts.size();
    if (f == 0) s->finished = true;
    *new_wins = f;
    return CR_OK;
}

int cr_solver_run(cr_solver* s, uint64_t* pass_counts, int32_t cap, int32_t* passes) {
    if (!s) return CR_ERR_INVALID;
    if (s->initialized && s->rules == CR_RULES_V1) {
        // two passes ahead with p = 1, whose passes are three launches; one with p > 1
        CR_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
        const size_t ahead = s->ctx->profiling ? 0 : (s->p == 1 ? 2 : 1);
        size_t stuck = 0;
        while (!s->finished && s->pass_counts.size() < (1 << 16)) {
            const size_t before = s->pass_counts.size();
            if (int rc = v1_advance(s, (1 << 16) - before, ahead)) return rc;
            stuck = s->pass_counts.size() == before ? stuck + 1 : 0;
            if (stuck > 4) return fail(s->ctx, CR_ERR_INTERNAL, "value slots kept overflowing");
        }
    }
    for (int i = 0; i < 1 << 16 && !s->finished; ++i) {
        uint64_t f;
        int rc = cr_solver_pass(s, &f);
        if (rc) return rc;
        if (s->finished) break;
    }
    if (!s->finished) return fail(s->ctx, CR_ERR_BUDGET, "no fixed point after 65536 passes");
    if (passes) *passes = (int32_t)s->pass_counts.size();
    if (pass_counts)
        for (size_t i = 0; i < s->pass_counts.size() && (int32_t)i < cap; ++i) pass_counts[i] = s->pass_counts[i];
    return CR_OK;
}

int cr_solver_verdict(cr_solver* s, cr_verdict* out) {
    if (!s || !out) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    CR_CUDA(ctx, cudaSetDevice(ctx->device));
    if (int rc = materialize_init(s)) return rc;
    cudaStream_t st = ctx->stream;
    unsigned long long* const d_key = s->d_ctl->counters + 1;
    unsigned long long* const h_key = s->kit.pinned + kHistRing;
    CR_CUDA(ctx, cudaMemsetAsync(d_key, 0xFF, sizeof(*d_key), st));
    if (s->rules == CR_RULES_V1) {
        V1Dev d = dev_view(s);
        launch_verdict(d, s->cols, d_key, s->grid_cop, st);
    } else {
        crgpu::v2_verdict(s->v2, d_key);
    }
    CR_CUDA(ctx, cudaGetLastError());
    CR_CUDA(ctx, cudaMemcpyAsync(h_key, d_key, sizeof(*h_key), cudaMemcpyDeviceToHost, st));
    CR_CUDA(ctx, cudaStreamSynchronize(st));
    s->unsynced = false;
    const unsigned long long key = *h_key;
    memset(out, 0, sizeof(*out));
    if (key == ~0ull || (int)(key >> 32) >= kMaxRound) {
        out->win = 0;
        out->best_config = -1;
        out->capture_plies = kMaxRound;
        return CR_OK;
    }
    out->win = 1;
    out->best_config = (int64_t)(key & 0xFFFFFFFFull);
    out->capture_plies = (int32_t)(key >> 32);
    // the configuration from its rank (as k_unrank): per position the largest vertex whose block of
    // configurations starts at or before it
    uint32_t rem = (uint32_t)out->best_config;
    int prev = 0;
    for (int i = 0; i < s->k; ++i) {
        const uint32_t* B = s->h_binom.data() + (size_t)i * (s->n + 1);
        int x = prev;
        while (x + 1 < s->n && B[x + 1] >= B[prev] - rem) ++x;
        rem -= B[prev] - B[x];
        out->positions[i] = (uint16_t)x;
        prev = x;
    }
    return CR_OK;
}

int cr_solver_sizes(cr_solver* s, cr_table_sizes* out) {
    if (!s || !out) return CR_ERR_INVALID;
    out->config_count = s->C;
    out->columns = s->cols;
    out->num_states = s->C * (uint64_t)s->n * s->cols;
    out->k = s->k;
    out->n = s->n;
    out->pad = 0;
    out->transitions = s->n_trans;
    return CR_OK;
}

int cr_solver_stats(cr_solver* s, cr_solve_stats* out) {
    if (!s || !out) return CR_ERR_INVALID;
    settle_init_time(s);
    *out = s->stats;
    uint64_t res = s->base_caps * (s->rules == CR_RULES_V1 ? 2 : 1);
    for (uint64_t c : s->pass_counts) res += c;
    out->resolved = res;
    return CR_OK;
}

int cr_solver_v2_hash_stats(cr_solver* s, cr_v2_hash_stats* out) {
    if (!s || !out) return CR_ERR_INVALID;
    *out = s->v2 ? crgpu::v2_hash_stats(s->v2) : cr_v2_hash_stats{};
    return CR_OK;
}

int cr_solver_set_forms(cr_solver* s, uint32_t mask) {
    if (!s) return CR_ERR_INVALID;
    if ((mask & ~CR_FORMS_ALL) || !(mask & (CR_FORM_PUSH | CR_FORM_PULL)))
        return fail(s->ctx, CR_ERR_INVALID, "forms: mask 0x%x (unknown bits, or neither push nor pull)", mask);
    if (s->rules != CR_RULES_V1 && mask != CR_FORMS_ALL)
        return fail(s->ctx, CR_ERR_INVALID, "forms: v2 solves have one form");
    if (mask == s->forms) return CR_OK;
    s->forms = mask;
    return CR_OK;
}

int cr_solver_set_v2_hash_capacity(cr_solver* s, uint64_t slots) {
    if (!s) return CR_ERR_INVALID;
    if (!s->v2) return CR_OK;   // v1 rules: no cloud table
    return crgpu::v2_set_hash_capacity(s->v2, slots, &s->ctx->err);
}

static const uint8_t* table_ptr(const cr_solver* s) {
    return s->rules == CR_RULES_V1 ? s->d_table : crgpu::v2_table(s->v2);
}

int cr_solver_digest(cr_solver* s, uint64_t* digest) {
    if (!s || !digest) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    CR_CUDA(ctx, cudaSetDevice(ctx->device));
    if (int rc = materialize_init(s)) return rc;
    cudaStream_t st = ctx->stream;
    unsigned long long* const d_sum = s->d_ctl->counters + 2;
    unsigned long long* const h_sum = s->kit.pinned + kHistRing + 1;
    CR_CUDA(ctx, cudaMemsetAsync(d_sum, 0, sizeof(*d_sum), st));
    launch_digest(table_ptr(s), s->C * (size_t)s->n * s->cols, d_sum, ctx->num_sms * 4, st);
    CR_CUDA(ctx, cudaGetLastError());
    CR_CUDA(ctx, cudaMemcpyAsync(h_sum, d_sum, sizeof(*h_sum), cudaMemcpyDeviceToHost, st));
    CR_CUDA(ctx, cudaStreamSynchronize(st));
    *digest = *h_sum;
    return CR_OK;
}

int cr_solver_device_states(cr_solver* s, void** dev_ptr, size_t* bytes) {
    if (!s || !dev_ptr || !bytes) return CR_ERR_INVALID;
    CR_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
    if (int rc = materialize_init(s)) return rc;
    s->shared = true;
    if (int rc = wait_for_table(s)) return rc;
    *dev_ptr = (void*)table_ptr(s);
    *bytes = s->C * (size_t)s->n * s->cols;
    return CR_OK;
}

int cr_solver_read_states(cr_solver* s, uint8_t* dst, size_t bytes) {
    if (!s || !dst) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    const size_t need = s->C * (size_t)s->n * s->cols;
    if (bytes < need) return fail(ctx, CR_ERR_INVALID, "states buffer holds %zu of %zu bytes", bytes, need);
    CR_CUDA(ctx, cudaSetDevice(ctx->device));
    if (int rc = materialize_init(s)) return rc;
    CR_CUDA(ctx, cudaMemcpyAsync(dst, table_ptr(s), need, cudaMemcpyDeviceToHost, ctx->stream));
    CR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return CR_OK;
}

int cr_solver_read_configs(cr_solver* s, uint8_t* dst, size_t bytes) {
    if (!s || !dst) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    if (s->n > 256) return fail(ctx, CR_ERR_LIMIT, "the table file stores vertices as uint8 (n <= 256)");
    const size_t cnt = s->C * (size_t)s->k;
    if (bytes < cnt) return fail(ctx, CR_ERR_INVALID, "configs buffer too small");
    std::vector<uint16_t> h(cnt);
    CR_CUDA(ctx, cudaMemcpyAsync(h.data(), s->d_configs, cnt * 2, cudaMemcpyDeviceToHost, ctx->stream));
    CR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (size_t i = 0; i < cnt; ++i) dst[i] = (uint8_t)h[i];
    return CR_OK;
}

int cr_solver_build_transitions(cr_solver* s, uint64_t* total) {
    if (!s) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    CR_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    if (!s->d_heads) {
        const int cap = trans_cap(s->k, s->cop_maxdeg);
        if (cap > 8192) return fail(ctx, CR_ERR_LIMIT, "successor fan-out %d too large for the CSR builder", cap);
        unsigned long long* counts = nullptr;
        CR_CUDA(ctx, get_or_shed(s, (void**)&counts, s->C * 8));
        CR_CUDA(ctx, get_or_shed(s, (void**)&s->d_heads, (s->C + 1) * 8));
        CR_CUDA(ctx, cudaMemsetAsync(&s->d_ctl->err, 0, sizeof(unsigned), st));
        const int grid = ctx->num_sms * 8;
        const uint32_t* trp = s->d_crp ? s->d_crp : s->d_rp;
        const uint16_t* tcol = s->d_ccol ? s->d_ccol : s->d_col;
        launch_trans(s->k, s->d_configs, (uint32_t)s->C, s->n, trp, tcol, s->d_binom, cap, counts,
                     nullptr, nullptr, &s->d_ctl->err, grid, st);
        launch_scan(counts, s->d_heads, (uint32_t)s->C, st);
        CR_CUDA(ctx, cudaGetLastError());
        unsigned long long tot = 0;
        CR_CUDA(ctx, cudaMemcpyAsync(&tot, s->d_heads + s->C, 8, cudaMemcpyDeviceToHost, st));
        CR_CUDA(ctx, cudaStreamSynchronize(st));
        ctx->cache.put(counts);
        s->n_trans = tot;
        CR_CUDA(ctx, get_or_shed(s, (void**)&s->d_trans, std::max<uint64_t>(tot, 1) * 8));
        launch_trans(s->k, s->d_configs, (uint32_t)s->C, s->n, trp, tcol, s->d_binom, cap, nullptr,
                     s->d_heads, s->d_trans, &s->d_ctl->err, grid, st);
        CR_CUDA(ctx, cudaGetLastError());
        unsigned bits = 0;
        int rc = check_err(s, &bits);
        if (rc) return rc;
        if (bits) return fail(ctx, CR_ERR_LIMIT, "successor fan-out exceeded the builder's buffer");
    }
    if (total) *total = s->n_trans;
    return CR_OK;
}

int cr_solver_perfect_game(cr_solver* s, int64_t* configs, int32_t* robbers, int32_t cap,
                           int32_t* count, int32_t* captured) {
    if (!s || !configs || !robbers || !count || !captured || cap <= 0) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    if (s->rules != CR_RULES_V1 || s->cols != 2 || s->cop_stay || s->robber_stay)
        return fail(ctx, CR_ERR_LIMIT, "the perfect game reads two-column (v1, p = 1) tables without stays");
    if (!s->finished) return fail(ctx, CR_ERR_STATE, "the solve has not reached its fixed point");
    *count = 0;
    *captured = 0;
    cr_verdict v;
    int rc = cr_solver_verdict(s, &v);
    if (rc) return rc;
    if (!v.win) return CR_OK;
    rc = cr_solver_build_transitions(s, nullptr);
    if (rc) return rc;
    cudaStream_t st = ctx->stream;
    long long* d_c = nullptr;
    int* d_r = nullptr;
    CR_CUDA(ctx, cudaMalloc(&d_c, sizeof(long long) * cap + sizeof(int) * (cap + 2)));
    d_r = reinterpret_cast<int*>(d_c + cap);
    launch_game(s->d_table, s->d_configs, s->d_heads, s->d_trans, s->d_rp, s->d_col, s->n, s->k,
                (long long)v.best_config, cap, d_c, d_r, d_r + cap, d_r + cap + 1, st);
    cudaError_t e = cudaGetLastError();
    int meta[2] = {0, 0};
    std::vector<long long> hc(cap);
    if (e == cudaSuccess) e = cudaMemcpyAsync(meta, d_r + cap, sizeof(meta), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(hc.data(), d_c, sizeof(long long) * cap, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(robbers, d_r, sizeof(int) * cap, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d_c);
    if (e != cudaSuccess) return fail(ctx, CR_ERR_CUDA, "perfect game: %s", cudaGetErrorString(e));
    for (int i = 0; i < meta[0] && i < cap; ++i) configs[i] = hc[i];
    *count = meta[0];
    *captured = meta[1];
    return CR_OK;
}

int cr_solver_read_transitions(cr_solver* s, uint64_t* heads, size_t heads_len, uint64_t* data,
                               size_t data_len) {
    if (!s) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    int rc = cr_solver_build_transitions(s, nullptr);
    if (rc) return rc;
    if (heads) {
        if (heads_len < s->C + 1) return fail(ctx, CR_ERR_INVALID, "heads buffer too small");
        CR_CUDA(ctx, cudaMemcpyAsync(heads, s->d_heads, (s->C + 1) * 8, cudaMemcpyDeviceToHost, ctx->stream));
    }
    if (data) {
        if (data_len < s->n_trans) return fail(ctx, CR_ERR_INVALID, "transitions buffer too small");
        if (s->n_trans) CR_CUDA(ctx, cudaMemcpyAsync(data, s->d_trans, s->n_trans * 8, cudaMemcpyDeviceToHost, ctx->stream));
    }
    CR_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return CR_OK;
}

int cr_solver_write_table_file(cr_solver* s, const char* path) {
    // CacheManager::saveAuxGraph (lib/include/CacheManager.h:28-75): 12 x u64 header
    // (k, N, columns, configCount, numStates, sizeof(T)=1, copSelf=0, robberSelf=0, four
    // section offsets), then configs u8, heads u64, transitions u64, states.
    if (!s || !path) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    int rc = cr_solver_build_transitions(s, nullptr);
    if (rc) return rc;
    const uint64_t cfg = s->C * (uint64_t)s->k, heads = (s->C + 1) * 8, trans = s->n_trans * 8;
    const uint64_t states = s->C * (uint64_t)s->n * s->cols;
    uint64_t hdr[12] = {(uint64_t)s->k, (uint64_t)s->n, (uint64_t)s->cols, s->C, states, 1,
                        (uint64_t)s->cop_stay, (uint64_t)s->robber_stay,
                        96, 96 + cfg, 96 + cfg + heads, 96 + cfg + heads + trans};
    FILE* f = fopen(path, "wb");
    if (!f) return fail(ctx, CR_ERR_IO, "cannot open %s for writing", path);
    std::vector<uint8_t> buf;
    bool ok = fwrite(hdr, 1, 96, f) == 96;
    buf.resize(cfg);
    rc = cr_solver_read_configs(s, buf.data(), buf.size());
    if (rc) { fclose(f); return rc; }
    ok = ok && fwrite(buf.data(), 1, cfg, f) == cfg;
    std::vector<uint64_t> hv(s->C + 1), tv(std::max<uint64_t>(s->n_trans, 1));
    rc = cr_solver_read_transitions(s, hv.data(), hv.size(), tv.data(), tv.size());
    if (rc) { fclose(f); return rc; }
    ok = ok && fwrite(hv.data(), 1, heads, f) == heads;
    ok = ok && (trans == 0 || fwrite(tv.data(), 1, trans, f) == trans);
    buf.resize(states);
    rc = cr_solver_read_states(s, buf.data(), buf.size());
    if (rc) { fclose(f); return rc; }
    ok = ok && fwrite(buf.data(), 1, states, f) == states;
    ok = (fclose(f) == 0) && ok;
    if (!ok) return fail(ctx, CR_ERR_IO, "short write to %s", path);
    return CR_OK;
}

int cr_solver_load_table_file(cr_solver* s, const char* path) {
    if (!s || !path) return CR_ERR_INVALID;
    cr_context* ctx = s->ctx;
    if (s->n > 256) return fail(ctx, CR_ERR_LIMIT, "the table file stores vertices as uint8 (n <= 256)");
    FILE* f = fopen(path, "rb");
    if (!f) return fail(ctx, CR_ERR_IO, "cannot open %s", path);
    std::vector<uint8_t> blob;
    {
        uint8_t buf[1 << 16];
        size_t got;
        while ((got = fread(buf, 1, sizeof(buf), f)) > 0) blob.insert(blob.end(), buf, buf + got);
        fclose(f);
    }
    if (blob.size() < 96) return fail(ctx, CR_ERR_IO, "%s: short header", path);
    uint64_t h[12];
    memcpy(h, blob.data(), 96);
    const uint64_t states = s->C * (uint64_t)s->n * s->cols;
    // the key fields (CacheManager.h:88-104): k, N, columns, configCount, numStates, the item
    // size and the self-edge rules
    if (h[0] != (uint64_t)s->k || h[1] != (uint64_t)s->n || h[2] != (uint64_t)s->cols || h[3] != s->C ||
        h[4] != states || h[5] != 1 || h[6] != (uint64_t)s->cop_stay || h[7] != (uint64_t)s->robber_stay)
        return fail(ctx, CR_ERR_INVALID, "%s was written for another solve", path);
    const uint64_t cfg = s->C * (uint64_t)s->k, heads = (s->C + 1) * 8;
    if (h[8] != 96 || h[9] != 96 + cfg || h[10] != h[9] + heads || h[11] < h[10] || (h[11] - h[10]) % 8 ||
        blob.size() != h[11] + states)
        return fail(ctx, CR_ERR_IO, "%s: sections do not match the header", path);
    std::vector<uint8_t> mine(cfg);
    int rc = cr_solver_read_configs(s, mine.data(), mine.size());
    if (rc) return rc;
    if (memcmp(mine.data(), blob.data() + h[8], cfg) != 0)
        return fail(ctx, CR_ERR_INVALID, "%s: configs section differs from this solver's", path);
    CR_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    const uint64_t ntrans = (h[11] - h[10]) / 8;
    if (!s->d_heads) CR_CUDA(ctx, get_or_shed(s, (void**)&s->d_heads, heads));
    if (s->d_trans && ntrans > s->n_trans) {
        ctx->cache.put(s->d_trans);
        s->d_trans = nullptr;
    }
    if (!s->d_trans) CR_CUDA(ctx, get_or_shed(s, (void**)&s->d_trans, std::max<uint64_t>(ntrans, 1) * 8));
    s->n_trans = ntrans;
    CR_CUDA(ctx, cudaMemcpyAsync(s->d_heads, blob.data() + h[9], heads, cudaMemcpyHostToDevice, st));
    if (ntrans) CR_CUDA(ctx, cudaMemcpyAsync(s->d_trans, blob.data() + h[10], ntrans * 8, cudaMemcpyHostToDevice, st));
    if (s->rules == CR_RULES_V2) {
        // the single-plane store of the v2 solver (k_cops_visibility_v2.cpp:170-182 loads the
        // same file layout with one column)
        if (int rc2 = crgpu::v2_load_states(s->v2, blob.data() + h[11], &ctx->err)) return rc2;
    } else {
        CR_CUDA(ctx, cudaMemcpyAsync(s->d_table, blob.data() + h[11], states, cudaMemcpyHostToDevice, st));
        launch_marks_from_table(s->d_table, (uint32_t)s->C, s->n, s->cols, s->rwp, s->d_marked, ctx->num_sms * 8, st);
        CR_CUDA(ctx, cudaGetLastError());
    }
    CR_CUDA(ctx, cudaStreamSynchronize(st));   // the host blob goes out of scope
    s->init_pending = false;
    s->initialized = true;
    s->finished = true;
    s->pass_counts.clear();
    return CR_OK;
}

int cr_solve(cr_context* ctx, const cr_graph* g, int32_t k, int32_t p, int32_t rules,
             uint8_t* states_out, size_t states_bytes, uint64_t* pass_counts, int32_t cap,
             int32_t* passes, cr_verdict* verdict, cr_solve_stats* stats) {
    cr_solver* s = nullptr;
    int rc = cr_solver_create(ctx, g, k, p, rules, &s);
    if (rc) return rc;
    rc = cr_solver_init(s, nullptr);
    if (!rc) rc = cr_solver_run(s, pass_counts, cap, passes);
    if (!rc && verdict) rc = cr_solver_verdict(s, verdict);
    if (!rc && states_out) rc = cr_solver_read_states(s, states_out, states_bytes);
    if (!rc && stats) rc = cr_solver_stats(s, stats);
    cr_solver_destroy(s);
    return rc;
}

}  // extern "C"
