// Context object: one GPU, one stream, optional NCCL communicator for sharded jobs.
#pragma once

#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"

namespace b200bpe {

struct NcclIdBlob { char bytes[128]; };

// NCCL entry points resolved at run time from the library the caller names, so that the
// process holds a single NCCL (the one its host framework already loaded).
struct NcclApi {
    void* handle = nullptr;
    int (*GetUniqueId)(void*) = nullptr;
    int (*CommInitRank)(void**, int, /*ncclUniqueId by value*/ NcclIdBlob, int) = nullptr;
    int (*CommDestroy)(void*) = nullptr;
    int (*AllReduce)(const void*, void*, size_t, int, int, void*, cudaStream_t) = nullptr;
    int (*AllGather)(const void*, void*, size_t, int, void*, cudaStream_t) = nullptr;
    int (*Send)(const void*, size_t, int, int, void*, cudaStream_t) = nullptr;
    int (*Recv)(void*, size_t, int, int, void*, cudaStream_t) = nullptr;
    int (*GroupStart)() = nullptr;
    int (*GroupEnd)() = nullptr;
    const char* (*GetErrorString)(int) = nullptr;
};
struct Ctx {
    std::atomic<uint32_t> holders{1};    // its creator, and every handle made with it
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t decode_stream = nullptr;   // the decoders': any thread may use it, and nobody records a graph from it
    int sm_count = 0;
    int cc = 0;
    int rank = 0, world = 1;
    NcclApi nccl;
    void* comm = nullptr;
    // Device memory of this context's short-lived objects, in the order of one of its streams: an allocation is a few microseconds when
    // the pool has the block, against hundreds for cudaMalloc.  At most POOL_KEEP bytes stay with the pool between calls; the
    // rest goes back to the device at the next synchronisation, and all of it with the context.  Blocks of more than POOL_BLOCK bytes are
    // not the pool's: it could not keep them, and maps and unmaps 10 GB in 50 ms each (at times ten times that), cudaMalloc and
    // cudaFree in 5 and 12.
    cudaMemPool_t pool = nullptr;
    static constexpr unsigned long long POOL_KEEP = 2ull << 30;
    static constexpr size_t POOL_BLOCK = 512ull << 20;
    std::vector<void*> large;
    std::mutex large_mutex;
    template <class T>
    cudaError_t alloc(T** p, size_t bytes, cudaStream_t on) {
        void* v = nullptr;
        cudaError_t e;
        if (bytes <= POOL_BLOCK) {
            e = cudaMallocFromPoolAsync(&v, bytes ? bytes : 1, pool, on);
        } else {
            e = cudaMalloc(&v, bytes);
            if (e == cudaErrorMemoryAllocation) {        // (what the pool keeps may be what is missing)
                cudaGetLastError();
                cudaStreamSynchronize(on);
                cudaMemPoolTrimTo(pool, 0);
                e = cudaMalloc(&v, bytes);
            }
            if (e == cudaSuccess) {
                std::lock_guard<std::mutex> lock(large_mutex);
                large.push_back(v);
            }
        }
        *p = static_cast<T*>(v);
        return e;
    }
    template <class T>
    cudaError_t alloc(T** p, size_t bytes) { return alloc(p, bytes, stream); }
    void free(void* p, cudaStream_t on) {
        if (!p) return;
        {
            std::unique_lock<std::mutex> lock(large_mutex);
            for (size_t i = 0; i < large.size(); i++)
                if (large[i] == p) {
                    large[i] = large.back();
                    large.pop_back();
                    lock.unlock();
                    cudaStreamSynchronize(on);           // (a pool's block may still be in use by what is enqueued; so may this one)
                    cudaFree(p);
                    return;
                }
        }
        cudaFreeAsync(p, on);
    }
    void free(void* p) { free(p, stream); }
    // Pinned host memory of this context's short-lived objects: cudaMallocHost takes 3 to 5 ms, half of a training call on a page of
    // text.  A few blocks are kept between objects, PINNED_KEEP bytes at most, and go with the context.  A block is only given back when no
    // copy to or from it is on its way.
    struct Pinned { void* p; size_t bytes; };
    std::vector<Pinned> pinned;
    std::mutex pinned_mutex;
    static constexpr size_t PINNED_KEEP = 4u << 20, PINNED_BLOCKS = 8;
    cudaError_t alloc_pinned(void** p, size_t* bytes) {     // *bytes: wanted, then what the block has
        {
            std::lock_guard<std::mutex> lock(pinned_mutex);
            for (size_t i = 0; i < pinned.size(); i++)
                if (pinned[i].bytes >= *bytes) {
                    *p = pinned[i].p;
                    *bytes = pinned[i].bytes;
                    pinned.erase(pinned.begin() + (ptrdiff_t)i);
                    return cudaSuccess;
                }
        }
        *bytes = (*bytes + 0xFFFFu) & ~(size_t)0xFFFFu;
        return cudaMallocHost(p, *bytes);
    }
    void free_pinned(void* p, size_t bytes) {
        if (!p) return;
        {
            std::lock_guard<std::mutex> lock(pinned_mutex);
            size_t kept = bytes;
            for (const Pinned& b : pinned) kept += b.bytes;
            if (pinned.size() < PINNED_BLOCKS && kept <= PINNED_KEEP) { pinned.push_back({p, bytes}); return; }
        }
        cudaFreeHost(p);
    }
};

// A handle's share of its context.  Handles give their memory back to the context's pool on its stream, so both stay until the last
// handle is gone, whichever order the caller destroys them in.  Declared first in a handle: it goes after everything else.
struct CtxHold {
    b200bpe_ctx* held = nullptr;
    void take(b200bpe_ctx* c);
    ~CtxHold();
};

b200bpe_status load_nccl(const char* path, NcclApi* api);

// Ask the L2 to keep [base, base + bytes) resident for the kernels launched on the context's
// stream from now on (a persisting access-policy window; captured graphs keep the window they
// were captured with).  The set-aside is capped, so a larger range is kept in proportion.
inline void set_persisting_window(Ctx* c, const void* base, size_t bytes) {
    int max_win = 0, max_persist = 0;
    cudaDeviceGetAttribute(&max_win, cudaDevAttrMaxAccessPolicyWindowSize, c->device);
    cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, c->device);
    const size_t want = bytes < (size_t)(max_win > 0 ? max_win : 0) ? bytes : (size_t)(max_win > 0 ? max_win : 0);
    if (want == 0 || max_persist <= 0) { cudaGetLastError(); return; }
    size_t set_aside = (size_t)max_persist;
    if (set_aside > ((size_t)64 << 20)) set_aside = (size_t)64 << 20;
    cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, set_aside);
    cudaStreamAttrValue attr{};
    attr.accessPolicyWindow.base_ptr = const_cast<void*>(base);
    attr.accessPolicyWindow.num_bytes = want;
    attr.accessPolicyWindow.hitRatio = want <= set_aside ? 1.0f : (float)set_aside / (float)want;
    attr.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    attr.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    cudaStreamSetAttribute(c->stream, cudaStreamAttributeAccessPolicyWindow, &attr);
    cudaGetLastError();
}

}  // namespace b200bpe

struct b200bpe_ctx { b200bpe::Ctx c; };
