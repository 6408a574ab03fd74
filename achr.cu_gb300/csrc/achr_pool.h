// Device workspaces of calls that own no context (the preconditioner's
// loss/gradient, coordinates, a GEMM's error word), from one memory pool per
// device.
//
// cudaMalloc and cudaFree of a call's fifteen buffers took 0.5 ms and stopped
// the device; the stream-ordered pool hands the same memory out again in about
// a microsecond.  It is the driver's pool object, so it is safe with any number
// of host threads and streams (memory freed on one stream is given to another
// only after the first stream's work), it keeps at most kKeepBytes between
// calls (anything above goes back at the next synchronisation), and it is
// destroyed with the process.
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <mutex>

namespace achr {

inline cudaError_t scratch_pool(cudaMemPool_t *pool) {
    constexpr unsigned long long kKeepBytes = 256ull << 20;
    static std::mutex mutex;
    static std::map<int, cudaMemPool_t> pools;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mutex);
    auto it = pools.find(dev);
    if (it == pools.end()) {
        cudaMemPoolProps p{};
        p.allocType = cudaMemAllocationTypePinned;
        p.location.type = cudaMemLocationTypeDevice;
        p.location.id = dev;
        cudaMemPool_t mp = nullptr;
        if ((e = cudaMemPoolCreate(&mp, &p)) != cudaSuccess) return e;
        unsigned long long keep = kKeepBytes;
        if ((e = cudaMemPoolSetAttribute(mp, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
            cudaMemPoolDestroy(mp);
            return e;
        }
        it = pools.emplace(dev, mp).first;
    }
    *pool = it->second;
    return cudaSuccess;
}

// One workspace for work on stream s; freed behind that work.
struct PoolBuf {
    char *p = nullptr;
    cudaStream_t s;
    explicit PoolBuf(cudaStream_t stream) : s(stream) {}
    PoolBuf(const PoolBuf &) = delete;
    PoolBuf &operator=(const PoolBuf &) = delete;
    ~PoolBuf() {
        if (p) cudaFreeAsync(p, s);
    }
    cudaError_t alloc(size_t bytes) {
        cudaMemPool_t pool;
        cudaError_t e = scratch_pool(&pool);
        if (e == cudaSuccess) e = cudaMallocFromPoolAsync(reinterpret_cast<void **>(&p), bytes ? bytes : 1, pool, s);
        if (e != cudaSuccess) p = nullptr;
        return e;
    }
};

}  // namespace achr
