// scratch.h -- short-lived device workspaces of the entry points that have no handle to keep them in.
//
// Each device has one stream-ordered memory pool of the library.  Memory that a call frees stays in
// the pool up to kScratchKeep bytes (the rest goes back to the device when a stream is next waited
// for), so that a repeated call does not map and unmap it again: cudaMallocAsync from the default
// pool, which keeps nothing, cost a forward projection 0.4 ms for a few KB and 1.4 ms for 68 MB.
// The pool orders reuse across streams and takes calls from any thread.
#pragma once
#include <algorithm>
#include <mutex>

#include "common.h"

namespace fdk {

constexpr unsigned long long kScratchKeep = 256ull << 20;

// The current device's pool, created at its first use.
inline int scratch_pool(cudaMemPool_t *out) {
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};
    int dev = 0;
    FDK_CUDA(cudaGetDevice(&dev));
    FDK_CHECK_ARG(dev < 64, "device %d", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!pools[dev]) {
        cudaMemPoolProps p{};
        p.allocType = cudaMemAllocationTypePinned;
        p.location.type = cudaMemLocationTypeDevice;
        p.location.id = dev;
        cudaMemPool_t pool = nullptr;
        FDK_CUDA(cudaMemPoolCreate(&pool, &p));
        unsigned long long keep = kScratchKeep;
        FDK_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        pools[dev] = pool;
    }
    *out = pools[dev];
    return FDK_OK;
}

// A workspace of the current device, ordered on st; returned to the pool on st by free() or the
// destructor.
struct Scratch {
    void *p = nullptr;
    cudaStream_t st = nullptr;
    int alloc(size_t bytes, cudaStream_t stream) {
        cudaMemPool_t pool = nullptr;
        FDK_TRY(scratch_pool(&pool));
        st = stream;
        FDK_CUDA(cudaMallocFromPoolAsync(&p, std::max<size_t>(bytes, 1), pool, stream));
        return FDK_OK;
    }
    int free() {
        void *q = p;
        p = nullptr;
        if (q) FDK_CUDA(cudaFreeAsync(q, st));
        return FDK_OK;
    }
    Scratch() = default;
    Scratch(const Scratch &) = delete;
    Scratch &operator=(const Scratch &) = delete;
    ~Scratch() {
        if (p) cudaFreeAsync(p, st);
    }
};

}  // namespace fdk
