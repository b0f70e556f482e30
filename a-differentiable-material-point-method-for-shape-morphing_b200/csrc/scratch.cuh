// scratch.cuh -- device scratch of the calls that hold no context (mesh sampling,
// surfaces): stream-ordered allocations on the default stream from a memory pool
// of the library's own, one per CUDA context.
//
// cudaMalloc and cudaFree of the 16-220 MB a call needs took 1-10 ms of 5-26 ms
// calls, unmapping above all.  The pool keeps at most kScratchKept bytes between
// calls (the driver returns the rest when the call's work is done) and gives
// those back too when an allocation of an engine or of a call fails
// (scratch_trim).  Pools are found by the context's unique id, so a context that
// was reset never meets an old one's pool; where no pool can be had the
// allocations are plain ones.  The driver's pools are safe to use from several
// threads, and all calls order their use on the same stream.  Nothing here throws:
// C entries use it bare.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <map>
#include <mutex>
#include <new>
#include <vector>

namespace dmpm_host {

constexpr unsigned long long kScratchKept = 256ull << 20;

struct ScratchPools {
    std::mutex m;
    std::map<unsigned long long, cudaMemPool_t> by_context;
};
inline ScratchPools& scratch_pools() {
    static ScratchPools p;
    return p;
}
// id of the calling thread's current context (the primary one, made if need be); 0: unknown
inline unsigned long long context_id() {
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static const GetId get = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return (GetId)f;
    }();
    if (!get || cudaFree(nullptr) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    unsigned long long id = 0;
    return get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}
inline cudaMemPool_t scratch_pool() {
    const unsigned long long id = context_id();
    if (id == 0) return nullptr;
    ScratchPools& p = scratch_pools();
    std::lock_guard<std::mutex> lock(p.m);
    auto it = p.by_context.find(id);
    if (it != p.by_context.end()) return it->second;
    try {
        it = p.by_context.emplace(id, nullptr).first;
    } catch (const std::bad_alloc&) {
        return nullptr;
    }
    cudaMemPool_t pool = nullptr;
    int dev = 0;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    unsigned long long keep = kScratchKept;
    if (cudaGetDevice(&dev) == cudaSuccess) {
        props.location.id = dev;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaGetLastError();
            pool = nullptr;
        }
    }
    it->second = pool;
    return pool;
}
// give back what the current context's pool keeps
inline void scratch_trim() {
    const unsigned long long id = context_id();
    ScratchPools& p = scratch_pools();
    std::lock_guard<std::mutex> lock(p.m);
    const auto it = p.by_context.find(id);
    if (it != p.by_context.end() && it->second) {
        cudaMemPoolTrimTo(it->second, 0);
        cudaGetLastError();
    }
}

// The device memory of one call, released when it goes.
class Scratch {
   public:
    Scratch() : pool_(scratch_pool()) {}
    Scratch(const Scratch&) = delete;
    Scratch& operator=(const Scratch&) = delete;
    ~Scratch() {
        for (const Block& b : blocks_) {
            if (b.pooled) cudaFreeAsync(b.p, nullptr);
            else cudaFree(b.p);
        }
    }
    // count elements and 32 bytes of padding, 256-byte aligned; null when there is no memory
    template <class T> T* alloc(size_t count) {
        const size_t bytes = count * sizeof(T) + 32;
        void* p = nullptr;
        try {
            blocks_.push_back({nullptr, false});
        } catch (const std::bad_alloc&) {
            return nullptr;
        }
        if (pool_ && cudaMallocFromPoolAsync(&p, bytes, pool_, nullptr) == cudaSuccess) {
            blocks_.back() = {p, true};
            return (T*)p;
        }
        cudaGetLastError();
        scratch_trim();
        if (cudaMalloc(&p, bytes) != cudaSuccess) {
            cudaGetLastError();
            blocks_.pop_back();
            return nullptr;
        }
        blocks_.back() = {p, false};
        return (T*)p;
    }

   private:
    struct Block {
        void* p;
        bool pooled;
    };
    cudaMemPool_t pool_;
    std::vector<Block> blocks_;
};

}  // namespace dmpm_host
