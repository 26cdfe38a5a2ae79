// scratch.h -- short-lived device workspaces of the entry points that have no handle to keep them in.
//
// Each context has one stream-ordered memory pool of the library.  Memory that a call frees stays in
// the pool up to kScratchKeep bytes (the rest goes back to the device when a stream is next waited
// for; fdk_scratch_trim gives back all of it), so that a repeated call does not map and unmap it again:
// cudaMallocAsync from the default pool, which keeps nothing, cost a forward projection 0.4 ms for a few
// KB and 1.4 ms for 68 MB.  The pool orders reuse across streams and takes calls from any thread.  A pool goes
// with its context (cudaDeviceReset): it is remembered with the context's id, which no later context has.
#pragma once
#include <cuda.h>

#include <algorithm>
#include <mutex>
#include <utility>
#include <vector>

#include "common.h"

namespace fdk {

constexpr unsigned long long kScratchKeep = 256ull << 20;

// The id of the calling thread's context (the primary one is created where there is none).  cuCtxGetId
// through the runtime's driver entry point: no libcuda link.
inline int context_id(unsigned long long *out) {
    using Fn = CUresult (*)(CUcontext, unsigned long long *);
    static const Fn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess;
        return ok && q == cudaDriverEntryPointSuccess ? reinterpret_cast<Fn>(p) : nullptr;
    }();
    if (fn && fn(nullptr, out) == CUDA_SUCCESS) return FDK_OK;
    FDK_CUDA(cudaFree(nullptr));  // makes one (not called where there is one: it would break a capture of another thread)
    if (!fn || fn(nullptr, out) != CUDA_SUCCESS) return fail(FDK_ERR_CUDA, "cuCtxGetId failed");
    return FDK_OK;
}

// The current context's pool, created at its first use; null if it has none and create is false.
inline int scratch_pool(cudaMemPool_t *out, bool create = true) {
    static std::mutex mu;
    static std::vector<std::pair<unsigned long long, cudaMemPool_t>> pools;  // (context id, pool)
    *out = nullptr;
    unsigned long long context = 0;
    FDK_TRY(context_id(&context));
    std::lock_guard<std::mutex> lock(mu);
    for (const auto &p : pools)
        if (p.first == context) *out = p.second;
    if (*out || !create) return FDK_OK;
    cudaMemPoolProps p{};
    p.allocType = cudaMemAllocationTypePinned;
    p.location.type = cudaMemLocationTypeDevice;
    FDK_CUDA(cudaGetDevice(&p.location.id));
    cudaMemPool_t pool = nullptr;
    FDK_CUDA(cudaMemPoolCreate(&pool, &p));
    unsigned long long keep = kScratchKeep;
    FDK_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    pools.emplace_back(context, pool);
    *out = pool;
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
