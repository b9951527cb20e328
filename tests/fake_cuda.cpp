// A CUDA runtime without a GPU, for tests of the library's host code: the library's
// own objects are linked against it.  Two devices with their own function attributes
// and multiprocessor counts, device memory in host memory, copies at once; a launch
// is checked for its dynamic shared memory and logged ("device grid kernel"), and a
// test's hook may play the kernel.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>

namespace {

struct State {
    std::recursive_mutex mu;
    std::map<const void *, std::string> names;
    std::map<std::pair<int, const void *>, int> smem;  // per device and function
    std::string log;
    std::map<cudaStream_t, cudaGraph_t> capturing;
    std::map<cudaGraph_t, std::pair<cudaHostFn_t, void *>> kept;  // a graph's user object
    int alloc_nodes = 0, pool_blocks = 0;                        // in graphs; from pools, not yet freed
};
State &state() {
    static State *s = new State();  // (kernels register before main, streams end after it)
    return *s;
}
thread_local int t_dev = 0;
thread_local cudaError_t t_err = cudaSuccess;
struct Call {
    dim3 grid, block;
    size_t smem;
    cudaStream_t st;
};
thread_local Call t_call;
void (*g_hook)(const char *, void **) = nullptr;

cudaError_t fail(cudaError_t e) { return t_err = e; }
cudaError_t launch(const void *fn, dim3 grid, size_t smem, void **args) {
    State &s = state();
    std::lock_guard<std::recursive_mutex> lk(s.mu);
    if (smem > 48 * 1024 && (int)smem > s.smem[{t_dev, fn}]) return fail(cudaErrorInvalidValue);
    s.log += std::to_string(t_dev) + " " + std::to_string(grid.x) + " " + s.names[fn] + "\n";
    if (g_hook) g_hook(s.names[fn].c_str(), args);
    return cudaSuccess;
}
cudaError_t memory(void **p, size_t n) { return (*p = std::calloc(1, n + 64)) ? cudaSuccess : fail(cudaErrorMemoryAllocation); }
int encode(void) { return 0; }  // cuTensorMapEncodeTiled: success

}  // namespace

extern "C" {

void fake_set_device(int dev) { t_dev = dev; }
void fake_set_hook(void (*hook)(const char *, void **)) { g_hook = hook; }
const char *fake_log() { return state().log.c_str(); }
void fake_clear() { state().log.clear(); }
int fake_alloc_nodes() { return state().alloc_nodes; }
int fake_pool_blocks() { return state().pool_blocks; }

void **__cudaRegisterFatBinary(void *) { return (void **)calloc(1, 8); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *fn, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
    state().names[fn] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st *st) {
    t_call = {g, b, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
    *g = t_call.grid;
    *b = t_call.block;
    *smem = t_call.smem;
    *(cudaStream_t *)st = t_call.st;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fn) {
    *k = (cudaKernel_t)fn;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void **args, size_t smem, cudaStream_t) {
    return launch((const void *)k, g, smem, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fn, void **args) {
    return launch(fn, c->gridDim, c->dynamicSmemBytes, args);
}
cudaError_t cudaFuncSetAttribute(const void *fn, enum cudaFuncAttribute, int v) {
    std::lock_guard<std::recursive_mutex> lk(state().mu);
    state().smem[{t_dev, fn}] = v;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = t_err;
    t_err = cudaSuccess;
    return e;
}
cudaError_t cudaGetDeviceCount(int *n) { return *n = 2, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = t_dev, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return t_dev = d, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr, int dev) { return *v = dev ? 7 : 5, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n) { return memory(p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return memory(p, n); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t st) {
    state().alloc_nodes += (int)state().capturing.count(st);
    ++state().pool_blocks;
    return memory(p, n);
}
cudaError_t cudaFree(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return --state().pool_blocks, std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return memory(p, n); }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { return *d = h, cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const struct cudaMemPoolProps *) { return memory((void **)p, 8); }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, enum cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *) {
    std::memset(a, 0, sizeof(*a));
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **, const void *) { return fail(cudaErrorInvalidSymbol); }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **fn, unsigned, unsigned long long,
                                             enum cudaDriverEntryPointQueryResult *r) {
    *fn = (void *)encode;
    *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, enum cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, enum cudaMemcpyKind, cudaStream_t) {
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, enum cudaMemcpyKind,
                              cudaStream_t) {
    for (size_t i = 0; i < h; ++i) std::memcpy((char *)d + i * dp, (const char *)s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return memory((void **)s, 8); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, enum cudaStreamCaptureMode) {
    return memory((void **)&state().capturing[s], 8);
}
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, enum cudaStreamCaptureStatus *st, unsigned long long *, cudaGraph_t *g,
                                     const cudaGraphNode_t **, const cudaGraphEdgeData **, size_t *) {
    const auto it = state().capturing.find(s);
    *st = it == state().capturing.end() ? cudaStreamCaptureStatusNone : cudaStreamCaptureStatusActive;
    if (g && it != state().capturing.end()) *g = it->second;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(enum cudaStreamCaptureMode *) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
    *g = state().capturing[s];
    state().capturing.erase(s);
    return cudaSuccess;
}
cudaError_t cudaUserObjectCreate(cudaUserObject_t *o, void *arg, cudaHostFn_t fn, unsigned, unsigned) {
    *o = (cudaUserObject_t) new std::pair<cudaHostFn_t, void *>(fn, arg);
    return cudaSuccess;
}
cudaError_t cudaUserObjectRelease(cudaUserObject_t o, unsigned) {
    auto *p = (std::pair<cudaHostFn_t, void *> *)o;
    p->first(p->second);
    delete p;
    return cudaSuccess;
}
cudaError_t cudaGraphRetainUserObject(cudaGraph_t g, cudaUserObject_t o, unsigned, unsigned) {
    auto *p = (std::pair<cudaHostFn_t, void *> *)o;
    state().kept[g] = *p;
    delete p;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    const auto it = state().kept.find(g);
    if (it != state().kept.end()) {
        const auto k = it->second;
        state().kept.erase(it);
        k.first(k.second);
    }
    return std::free(g), cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { return memory((void **)e, 8); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return memory((void **)e, 8); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }

}  // extern "C"
