// lla_scratch.cpp -- see lla_scratch.h.
#include "lla_scratch.h"

#include <mutex>
#include <vector>

#include "lla_device.h"

namespace lla {

// One device's pool, the stream that allocations beside a capture are ordered on, and
// the blocks that graphs have handed back.
struct DevicePool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t side = nullptr;
    std::vector<void *> back;
};
static std::mutex g_mu;       // pools and streams
static std::mutex g_back_mu;  // the lists of blocks handed back (no CUDA call under it)
// (never destroyed: a graph may outlive this file's statics)
static DevicePool *const g_pools = new DevicePool[kMaxDevices];

static cudaError_t current_device(int *dev) {
    const cudaError_t e = cudaGetDevice(dev);
    if (e != cudaSuccess) return e;
    return *dev >= 0 && *dev < kMaxDevices ? cudaSuccess : cudaErrorInvalidDevice;
}

// The current device's pool, created on the first call there; with g_mu held.
static cudaError_t device_pool(DevicePool &d, int dev) {
    cudaError_t e;
    if (!d.pool) {
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
        d.pool = p;
    }
    std::vector<void *> back;
    {
        std::lock_guard<std::mutex> lk(g_back_mu);
        back.swap(d.back);
    }
    for (void *p : back) cudaFreeAsync(p, d.side);
    return cudaSuccess;
}

struct GraphBlock {
    int dev;
    void *p;
};

// The last graph that used the block is gone.  Called by the driver, which allows no
// CUDA call here.
static void CUDART_CB graph_block_back(void *arg) {
    GraphBlock *b = (GraphBlock *)arg;
    {
        std::lock_guard<std::mutex> lk(g_back_mu);
        g_pools[b->dev].back.push_back(b->p);
    }
    delete b;
}

// A block for a launch sequence that is captured into `graph`, which keeps it.
static cudaError_t alloc_for_graph(size_t bytes, cudaGraph_t graph, void **out) {
    int dev = 0;
    cudaError_t e = current_device(&dev);
    if (e != cudaSuccess) return e;
    cudaStream_t side = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        DevicePool &d = g_pools[dev];
        if (!d.side && (e = cudaStreamCreateWithFlags(&d.side, cudaStreamNonBlocking)) != cudaSuccess) {
            d.side = nullptr;
            return e;
        }
        if ((e = device_pool(d, dev)) != cudaSuccess) return e;
        side = d.side;
        if ((e = cudaMallocFromPoolAsync(out, bytes, d.pool, side)) != cudaSuccess) return e;
    }
    if ((e = cudaStreamSynchronize(side)) == cudaSuccess) {  // allocated before any launch of the graph
        GraphBlock *b = new GraphBlock{dev, *out};
        cudaUserObject_t obj = nullptr;
        e = cudaUserObjectCreate(&obj, b, graph_block_back, 1, cudaUserObjectNoDestructorSync);
        if (e != cudaSuccess) {
            delete b;
        } else {
            e = cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove);
            if (e == cudaSuccess) return cudaSuccess;
            cudaUserObjectRelease(obj, 1);  // hands the block back
            return e;
        }
    }
    cudaFreeAsync(*out, side);
    return e;
}

cudaError_t StreamScratch::alloc(size_t bytes) {
    bytes = bytes > 0 ? bytes : 1;
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamGetCaptureInfo(st_, &status, nullptr, &graph);
    if (e != cudaSuccess) return e;
    if (status != cudaStreamCaptureStatusNone) {
        // the calls below concern another stream, which a capture forbids unless it is relaxed
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        if ((e = cudaThreadExchangeStreamCaptureMode(&mode)) != cudaSuccess) return e;
        e = status == cudaStreamCaptureStatusActive ? alloc_for_graph(bytes, graph, &p_)
                                                    : cudaErrorStreamCaptureInvalidated;
        cudaThreadExchangeStreamCaptureMode(&mode);
        kept_by_graph_ = true;
    } else {
        int dev = 0;
        if ((e = current_device(&dev)) != cudaSuccess) return e;
        std::lock_guard<std::mutex> lk(g_mu);
        if ((e = device_pool(g_pools[dev], dev)) == cudaSuccess)
            e = cudaMallocFromPoolAsync(&p_, bytes, g_pools[dev].pool, st_);
    }
    if (e != cudaSuccess) p_ = nullptr;
    return e;
}

}  // namespace lla
