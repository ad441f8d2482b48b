// crgpu_ctx.h - the context object behind the C ABI (shared by the API translation units).
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

// Device blocks a context keeps after the solver that used them is destroyed, so that the next
// solve of a similar size on the same context (the one-call cr_solve in a loop, a solve server's
// worker) takes them instead of calling cudaMalloc and cudaFree, which map and unmap pages and
// synchronise the device.  The free blocks are held up to `limit` bytes (the largest go first); a
// block is reused for a request of at least two thirds of its size, and requests below 1 MiB are
// rounded up to a power of two so that small solves of different sizes share theirs.  Reuse is
// ordered by the context's stream, the only stream its solvers use; blocks come back only from
// destroyed solvers, all of whose work is on that stream.  A solver may be destroyed from another
// thread than the one solving on the context (a solve server's client releasing a table), so the
// cache takes a lock.
struct cr_block_cache {
    static constexpr size_t kSmallBytes = 1u << 20;
    struct Block {
        void* p;
        size_t bytes;
    };
    std::vector<Block> held;                     // free
    std::unordered_map<void*, size_t> used;
    size_t held_bytes = 0, used_bytes = 0, peak_used = 0;
    size_t limit = 4ull << 30;
    size_t most = ~size_t(0);                    // of held and used blocks together (a full device, for tests)
    std::mutex mu;

    cudaError_t get(void** out, size_t bytes) {
        std::lock_guard<std::mutex> lock(mu);
        *out = nullptr;
        if (bytes < kSmallBytes) {
            size_t b = 512;
            while (b < bytes) b <<= 1;
            bytes = b;
        }
        int best = -1;
        for (int i = 0; i < (int)held.size(); ++i) {
            const Block& b = held[i];
            if (b.bytes >= bytes && b.bytes - bytes <= bytes / 2 && (best < 0 || b.bytes < held[best].bytes)) best = i;
        }
        if (best >= 0) {
            *out = held[best].p;
            used[held[best].p] = held[best].bytes;
            held_bytes -= held[best].bytes;
            add_used(held[best].bytes);
            held[best] = held.back();
            held.pop_back();
            return cudaSuccess;
        }
        cudaError_t e = allocate(out, bytes);
        if (e == cudaErrorMemoryAllocation) {   // give the held blocks back and try once more
            release_free();
            e = allocate(out, bytes);
        }
        if (e != cudaSuccess) return e;
        used[*out] = bytes;
        add_used(bytes);
        return cudaSuccess;
    }
    void put(void* p) {
        if (!p) return;
        std::lock_guard<std::mutex> lock(mu);
        const auto it = used.find(p);
        if (it == used.end()) {
            cudaFree(p);
            return;
        }
        held.push_back(Block{p, it->second});
        held_bytes += it->second;
        used_bytes -= it->second;
        used.erase(it);
        trim();
    }
    void set_limit(size_t bytes) {
        std::lock_guard<std::mutex> lock(mu);
        limit = bytes;
        trim();
    }
    void clear() {
        std::lock_guard<std::mutex> lock(mu);
        release_free();
    }
    size_t free_bytes() {
        std::lock_guard<std::mutex> lock(mu);
        return held_bytes;
    }
    // (the callers below hold the lock)
    void add_used(size_t bytes) {
        used_bytes += bytes;
        if (used_bytes > peak_used) peak_used = used_bytes;
    }
    // An error is the caller's to report: none is left behind for the check of a later launch.
    cudaError_t allocate(void** out, size_t bytes) {
        if (bytes > most || held_bytes + used_bytes > most - bytes) return cudaErrorMemoryAllocation;
        const cudaError_t e = cudaMalloc(out, bytes);
        if (e != cudaSuccess) {
            *out = nullptr;
            cudaGetLastError();
        }
        return e;
    }
    void trim() {
        while (held_bytes > limit) {
            size_t big = 0;
            for (size_t i = 1; i < held.size(); ++i)
                if (held[i].bytes > held[big].bytes) big = i;
            cudaFree(held[big].p);
            held_bytes -= held[big].bytes;
            held[big] = held.back();
            held.pop_back();
        }
    }
    void release_free() {
        for (const Block& b : held) cudaFree(b.p);
        held.clear();
        held_bytes = 0;
    }
};

// What every solver needs besides device memory: a pinned read-back area and timing events.  The
// context keeps a few for the next solvers (pinning a page and freeing it cost more than a small
// solve).
struct cr_solver_kit {
    static constexpr int kWords = 128;           // unsigned long long
    unsigned long long* pinned = nullptr;
    cudaEvent_t ev[4] = {};

    cudaError_t make() {
        cudaError_t e = cudaMallocHost(&pinned, kWords * sizeof(unsigned long long));
        for (int i = 0; i < 4 && e == cudaSuccess; ++i) e = cudaEventCreate(&ev[i]);
        return e;
    }
    void release() {
        if (pinned) cudaFreeHost(pinned);
        for (cudaEvent_t e : ev)
            if (e) cudaEventDestroy(e);
        *this = cr_solver_kit{};
    }
};

struct cr_context {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int num_sms = 1;
    bool profiling = false;
    std::string err;
    cr_block_cache cache;
    static constexpr size_t kMaxKits = 8;
    std::vector<cr_solver_kit> kits;
    std::mutex kits_mu;

    cudaError_t get_kit(cr_solver_kit* out) {
        {
            std::lock_guard<std::mutex> lock(kits_mu);
            if (!kits.empty()) {
                *out = kits.back();
                kits.pop_back();
                return cudaSuccess;
            }
        }
        const cudaError_t e = out->make();
        if (e != cudaSuccess) out->release();
        return e;
    }
    void put_kit(cr_solver_kit kit) {
        if (!kit.pinned) return;
        {
            std::lock_guard<std::mutex> lock(kits_mu);
            if (kits.size() < kMaxKits) {
                kits.push_back(kit);
                return;
            }
        }
        kit.release();
    }
};
