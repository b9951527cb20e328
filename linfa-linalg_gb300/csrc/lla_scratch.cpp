// lla_scratch.cpp -- see lla_scratch.h.
#include "lla_scratch.h"

#include "lla_device.h"

#include <mutex>

namespace lla {

static std::mutex g_pool_mu;
static cudaMemPool_t g_pool[kMaxDevices] = {};

// The current device's pool, created on the first call there.
static cudaError_t device_pool(cudaMemPool_t *out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (!g_pool[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t p = nullptr;
        if ((e = cudaMemPoolCreate(&p, &props)) != cudaSuccess) return e;
        unsigned long long keep = kScratchKeepBytes;
        if ((e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
            cudaMemPoolDestroy(p);
            return e;
        }
        g_pool[dev] = p;
    }
    *out = g_pool[dev];
    return cudaSuccess;
}

cudaError_t StreamScratch::alloc(size_t bytes) {
    cudaMemPool_t pool = nullptr;
    cudaError_t e = device_pool(&pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&p_, bytes > 0 ? bytes : 1, pool, st_);
    if (e != cudaSuccess) p_ = nullptr;
    return e;
}

}  // namespace lla
