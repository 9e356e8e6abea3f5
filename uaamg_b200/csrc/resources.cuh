// resources.cuh -- per-device pools that make solver handles cheap to create.
//
// A FLIP substep builds a new hierarchy for every pressure solve
// (FLIP_vdb.cpp:3132-3141), so the fixed cost of a handle matters as much as
// the solve.  cudaMalloc/cudaFree, pinned host allocation and stream creation
// each cost tens of microseconds to milliseconds and synchronise the device,
// so handles draw all three from per-device pools instead:
//  * device memory: a private stream-ordered memory pool whose release
//    threshold is "never", so freed blocks are reused without OS calls, and a
//    bounded list of freed blocks in front of it (ctx_dev_alloc): a handle's
//    60 allocations took 12 ms from the pool alone in a process that had used
//    120 handles (each one's streams leave freed blocks the pool looks
//    through), against 0.2 ms in a fresh one;
//  * streams and pinned host blocks: free lists.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <unordered_set>
#include <utility>
#include <vector>

namespace uaamg {

// A freed device block: for any later use (every use of it has ended), or for
// use in the order of the stream it was freed on.
struct FreeBlock {
    void* p;
    size_t cap;
    cudaStream_t s;
    bool idle;
};
constexpr size_t FREE_BLOCKS_BYTES = size_t(2) << 30;  // kept per device at most
constexpr size_t FREE_BLOCKS_MAX = 512;

struct DeviceCtx {
    int device = -1;
    int sms = 0;  // streaming multiprocessors of the device
    cudaMemPool_t pool = nullptr;
    std::mutex mu;
    std::vector<cudaStream_t> streams;
    std::unordered_set<cudaStream_t> own_streams;  // every stream made here; they are never destroyed
    std::vector<std::pair<size_t, void*>> pinned;  // free pinned blocks (capacity, pointer)
    std::vector<cudaStream_t> capturing;           // streams being captured into the library's own graphs (CaptureMark)
    cudaStream_t free_stream = nullptr;            // where idle blocks of no usable stream go back; nothing else runs there
    std::unordered_map<void*, size_t> live;        // capacity of the blocks in use that may go to `blocks`
    std::vector<FreeBlock> blocks;                 // freed blocks, oldest first
    size_t blocks_bytes = 0;
};

inline std::mutex& ctx_registry_mutex() {
    static std::mutex m;
    return m;
}

// Context of the current device (created on first use).
inline DeviceCtx* device_ctx(cudaError_t* err) {
    static DeviceCtx* ctxs[64] = {nullptr};
    int dev = 0;
    *err = cudaGetDevice(&dev);
    if (*err != cudaSuccess) return nullptr;
    if (dev < 0 || dev >= 64) { *err = cudaErrorInvalidDevice; return nullptr; }
    std::lock_guard<std::mutex> lk(ctx_registry_mutex());
    if (!ctxs[dev]) {
        DeviceCtx* c = new DeviceCtx();
        c->device = dev;
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        *err = cudaMemPoolCreate(&c->pool, &props);
        if (*err != cudaSuccess) { delete c; return nullptr; }
        uint64_t thr = UINT64_MAX;
        *err = cudaMemPoolSetAttribute(c->pool, cudaMemPoolAttrReleaseThreshold, &thr);
        if (*err != cudaSuccess) { delete c; return nullptr; }
        *err = cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, dev);
        if (*err != cudaSuccess) { delete c; return nullptr; }
        *err = cudaStreamCreateWithFlags(&c->free_stream, cudaStreamNonBlocking);
        if (*err != cudaSuccess) { delete c; return nullptr; }
        ctxs[dev] = c;
    }
    return ctxs[dev];
}

inline cudaError_t ctx_stream_acquire(DeviceCtx* c, cudaStream_t* s) {
    {
        std::lock_guard<std::mutex> lk(c->mu);
        if (!c->streams.empty()) {
            *s = c->streams.back();
            c->streams.pop_back();
            return cudaSuccess;
        }
    }
    const cudaError_t e = cudaStreamCreateWithFlags(s, cudaStreamNonBlocking);
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> lk(c->mu);
        c->own_streams.insert(*s);
    }
    return e;
}
inline void ctx_stream_release(DeviceCtx* c, cudaStream_t s) {
    if (!s) return;
    std::lock_guard<std::mutex> lk(c->mu);
    c->streams.push_back(s);
}

// pinned host block of at least `bytes`; *cap receives its capacity
inline cudaError_t ctx_pinned_acquire(DeviceCtx* c, size_t bytes, void** p, size_t* cap) {
    {
        std::lock_guard<std::mutex> lk(c->mu);
        size_t best = (size_t)-1;
        int bi = -1;
        for (size_t i = 0; i < c->pinned.size(); ++i)
            if (c->pinned[i].first >= bytes && c->pinned[i].first < best) { best = c->pinned[i].first; bi = (int)i; }
        if (bi >= 0) {
            *cap = c->pinned[bi].first;
            *p = c->pinned[bi].second;
            c->pinned.erase(c->pinned.begin() + bi);
            return cudaSuccess;
        }
    }
    size_t sz = 4096;
    while (sz < bytes) sz <<= 1;
    *cap = sz;
    return cudaMallocHost(p, sz);
}
inline void ctx_pinned_release(DeviceCtx* c, void* p, size_t cap) {
    if (!p) return;
    std::lock_guard<std::mutex> lk(c->mu);
    c->pinned.push_back({cap, p});
}

// Device memory.  A block freed on one of the context's own streams (or the
// legacy default stream) is kept for later allocations on that stream, in
// whose order its reuse is; a block freed as idle for any stream.  Other
// streams are a caller's, who may destroy them: their frees, and all of a
// capturing stream's, go to the pool.  At most FREE_BLOCKS_BYTES are kept
// (the oldest go back to the pool), none when an allocation fails.  A kept
// block goes back on the stream it was freed on, where the pool can reuse it at
// once.  While that stream is being captured it must not (another thread's
// graph would take the free in, fail or repeat it): an idle block then goes
// back on free_stream, any other stays.
inline size_t dev_block_size(size_t bytes) {  // classes 1/8 of a power of two apart, so that similar sizes share blocks
    if (bytes < 1024) return 1024;
    if (bytes > (size_t(64) << 20)) return (bytes + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1);
    size_t step = 128;
    while (step * 16 <= bytes) step <<= 1;
    return (bytes + step - 1) & ~(step - 1);
}
inline bool ctx_capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return st != cudaStreamCaptureStatusNone;
}
// A stream that is about to be captured into a graph of the library, until the capture has ended.
struct CaptureMark {
    DeviceCtx* c;
    cudaStream_t s;
    CaptureMark(DeviceCtx* ctx, cudaStream_t st) : c(ctx), s(st) {
        std::lock_guard<std::mutex> lk(c->mu);
        c->capturing.push_back(s);
    }
    CaptureMark(const CaptureMark&) = delete;
    CaptureMark& operator=(const CaptureMark&) = delete;
    ~CaptureMark() {
        std::lock_guard<std::mutex> lk(c->mu);
        c->capturing.erase(std::find(c->capturing.begin(), c->capturing.end(), s));
    }
};
// Gives the oldest kept blocks back to the pool until at most `bytes` in `count` blocks are left; c->mu is held (so that
// no capture starts meanwhile).  used: receives the streams they were freed on.
inline cudaError_t ctx_dev_give_back(DeviceCtx* c, size_t bytes, size_t count, std::vector<cudaStream_t>* used = nullptr) {
    if (c->blocks_bytes <= bytes && c->blocks.size() <= count) return cudaSuccess;
    cudaError_t e = cudaSuccess;
    size_t left = c->blocks.size(), w = 0;
    for (size_t i = 0; i < c->blocks.size(); ++i) {
        FreeBlock b = c->blocks[i];
        bool keep = c->blocks_bytes <= bytes && left <= count;
        if (!keep && (std::find(c->capturing.begin(), c->capturing.end(), b.s) != c->capturing.end() || ctx_capturing(b.s))) {
            if (b.idle) b.s = c->free_stream;
            else keep = true;
        }
        if (keep) {
            c->blocks[w++] = b;
            continue;
        }
        const cudaError_t q = cudaFreeAsync(b.p, b.s);
        if (q != cudaSuccess) e = q;
        c->blocks_bytes -= b.cap;
        --left;
        if (used && std::find(used->begin(), used->end(), b.s) == used->end()) used->push_back(b.s);
    }
    c->blocks.resize(w);
    return e;
}
inline cudaError_t ctx_dev_alloc(DeviceCtx* c, void** p, size_t bytes, cudaStream_t s) {
    const size_t cap = dev_block_size(bytes);
    const bool plain = ctx_capturing(s);
    if (!plain) {
        std::lock_guard<std::mutex> lk(c->mu);
        size_t best = c->blocks.size();
        for (size_t i = c->blocks.size(); i-- > 0;) {  // the newest of the best fits
            const FreeBlock& b = c->blocks[i];
            if (b.cap < cap || b.cap > cap + cap / 4 || !(b.idle || b.s == s)) continue;
            if (best == c->blocks.size() || b.cap < c->blocks[best].cap) best = i;
        }
        if (best < c->blocks.size()) {
            *p = c->blocks[best].p;
            c->live[*p] = c->blocks[best].cap;
            c->blocks_bytes -= c->blocks[best].cap;
            c->blocks.erase(c->blocks.begin() + (ptrdiff_t)best);
            return cudaSuccess;
        }
    }
    cudaError_t e = cudaMallocFromPoolAsync(p, cap, c->pool, s);
    if (e == cudaErrorMemoryAllocation && !plain) {
        cudaGetLastError();
        {
            std::lock_guard<std::mutex> lk(c->mu);
            std::vector<cudaStream_t> used;
            ctx_dev_give_back(c, 0, 0, &used);
            for (cudaStream_t u : used) cudaStreamSynchronize(u);
        }
        e = cudaMallocFromPoolAsync(p, cap, c->pool, s);
    }
    if (e == cudaSuccess && !plain) {
        std::lock_guard<std::mutex> lk(c->mu);
        c->live[*p] = cap;
    }
    return e;
}
// whether a stream has nothing left to do
inline bool ctx_stream_idle(cudaStream_t s) {
    const cudaError_t e = cudaStreamQuery(s);
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
}
// idle: every use of the block, on whatever stream, has ended
inline cudaError_t ctx_dev_free(DeviceCtx* c, void* p, cudaStream_t s, bool idle = false) {
    if (!p) return cudaSuccess;
    const bool capturing = ctx_capturing(s);
    {
        std::lock_guard<std::mutex> lk(c->mu);
        const auto it = c->live.find(p);
        const size_t cap = it == c->live.end() ? 0 : it->second;
        if (cap) c->live.erase(it);
        const bool own = s == nullptr || c->own_streams.count(s) != 0;
        if (cap && cap <= FREE_BLOCKS_BYTES / 4 && !capturing && (own || idle)) {
            c->blocks.push_back({p, cap, own ? s : c->free_stream, idle});
            c->blocks_bytes += cap;
            return ctx_dev_give_back(c, FREE_BLOCKS_BYTES, FREE_BLOCKS_MAX);
        }
    }
    return cudaFreeAsync(p, s);
}

}  // namespace uaamg
