// A CUDA runtime without a device, linked in place of the real one: device memory is host memory,
// copies and fills are checked against its blocks, kernels do not run.  A hook sees every launch (and
// may write what the kernel would have), any call can be made to fail, and memory can be limited.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<uintptr_t, size_t> blocks;
std::map<const void *, std::string> kernels;
std::map<const void *, std::pair<void *, size_t>> vars;
std::map<std::string, std::pair<int, int>> fails;  // call or kernel -> calls until it fails, error
std::string launched;
size_t limit = ~size_t(0), used = 0, largest = 0;
int last = 0, stray = 0;
int (*hook)(const char *, void **) = nullptr;
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
cudaStream_t cfg_stream;

cudaError_t done(int e) {
    if (e) last = e;
    return (cudaError_t)e;
}
int failing(const std::string &name) {
    for (auto &f : fails)
        if (name.find(f.first) != std::string::npos && f.second.first-- == 0) return f.second.second;
    return 0;
}
bool device(const void *p, size_t n) {
    auto it = blocks.upper_bound((uintptr_t)p);
    if (it == blocks.begin()) return false;
    --it;
    return (uintptr_t)p + n <= it->first + it->second;
}
int check(const void *p, size_t n) {
    if (n == 0 || device(p, n)) return 0;
    ++stray;
    return cudaErrorInvalidValue;
}
}  // namespace

#define OK(name, args) \
    cudaError_t name args { return done(failing(#name)); }

extern "C" {
void fake_reset() {
    fails.clear();
    launched.clear();
    limit = ~size_t(0);
    largest = 0;
    last = stray = 0;
    hook = nullptr;
}
void fake_hook(int (*h)(const char *, void **)) { hook = h; }
void fake_fail(const char *name, int after, int code) { fails[name] = {after, code}; }
void fake_limit(size_t bytes) { limit = bytes; }
size_t fake_used() { return used; }
size_t fake_largest() { return largest; }
int fake_stray() { return stray; }
const char *fake_launched() { return launched.c_str(); }
void *fake_alloc(size_t n) {
    void *p = nullptr;
    cudaMalloc(&p, n);
    return p;
}

cudaError_t cudaMalloc(void **p, size_t n) {
    const int e = failing("cudaMalloc");
    if (e) return done(e);
    if (n > limit || used > limit - n) return done(cudaErrorMemoryAllocation);
    *p = std::calloc(1, n ? n : 1);
    blocks[(uintptr_t)*p] = n;
    used += n;
    largest = n > largest ? n : largest;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (!p) return cudaSuccess;
    auto it = blocks.find((uintptr_t)p);
    if (it == blocks.end()) {
        ++stray;
        return done(cudaErrorInvalidValue);
    }
    used -= it->second;
    blocks.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return *p = std::calloc(1, n), cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { return *p = std::calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
    int e = failing("cudaMemcpy");
    if (!e && (k == cudaMemcpyHostToDevice || k == cudaMemcpyDeviceToDevice)) e = check(d, n);
    if (!e && (k == cudaMemcpyDeviceToHost || k == cudaMemcpyDeviceToDevice)) e = check(s, n);
    if (e) return done(e);
    if (n) std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) {
    int e = failing("cudaMemsetAsync");
    if (!e) e = check(d, n);
    if (e) return done(e);
    if (n) std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::memset(a, 0, sizeof *a);
    a->type = device(p, 1) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const int e = last;
    last = 0;
    return (cudaError_t)e;
}
cudaError_t cudaPeekAtLastError() { return (cudaError_t)last; }
const char *cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount           ? 148
         : a == cudaDevAttrL2CacheSize                 ? 126 << 20
         : a == cudaDevAttrComputeCapabilityMajor      ? 10
         : a == cudaDevAttrMaxGridDimX                 ? 2147483647
         : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448
                                                       : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp *p, int) {
    std::memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = 148;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    std::memset(a, 0, sizeof *a);
    a->ptxVersion = a->binaryVersion = 100;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int v) {
    const int e = failing("cudaFuncSetAttribute");
    return done(e ? e : v > 232448 ? cudaErrorInvalidValue : 0);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int threads, size_t smem, unsigned) {
    const int a = 2048 / threads, b = (int)(233472 / (smem + 1024));
    return *n = a < b ? a : b, cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int threads, size_t smem) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, threads, smem, 0);
    *n = *n < 3 ? *n : 3;  // the scorers' launch bounds
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *s) {
    auto &v = vars[s];
    if (!v.first) cudaMalloc(&v.first, v.second);
    return *p = v.first, cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **args, size_t smem, cudaStream_t) {
    const std::string &name = kernels[f];
    int e = failing(name);
    if (!e && (g.x < 1 || g.y < 1 || g.z < 1 || g.y > 65535 || g.z > 65535 || b.x * b.y * b.z > 1024 || smem > 232448))
        e = cudaErrorInvalidConfiguration;
    if (e) return done(e);
    launched += name + "\n";
    return done(hook ? hook(name.c_str(), args) : 0);
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, cudaStream_t st) {
    cfg_grid = g, cfg_block = b, cfg_smem = s, cfg_stream = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
    *g = cfg_grid, *b = cfg_block, *s = cfg_smem, *(cudaStream_t *)st = cfg_stream;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *f, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
    kernels[f] = name;
}
void __cudaRegisterVar(void **, char *v, char *, const char *, int, size_t n, int, int) { vars[v] = {nullptr, n}; }
OK(cudaSetDevice, (int))
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = (cudaStream_t)1, cudaSuccess; }
OK(cudaStreamDestroy, (cudaStream_t))
OK(cudaStreamSynchronize, (cudaStream_t))
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)1, cudaSuccess; }
OK(cudaEventDestroy, (cudaEvent_t))
OK(cudaEventRecord, (cudaEvent_t, cudaStream_t))
OK(cudaEventSynchronize, (cudaEvent_t))
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return done(cudaErrorNotSupported); }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t *, const cudaGraphEdgeData *, size_t,
                                          cudaStreamCaptureMode) {
    return done(cudaErrorNotSupported);
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return done(cudaErrorNotSupported); }
cudaError_t cudaGraphAddNode(cudaGraphNode_t *, cudaGraph_t, const cudaGraphNode_t *, size_t, cudaGraphNodeParams *) {
    return done(cudaErrorNotSupported);
}
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle *, cudaGraph_t, unsigned, unsigned) {
    return done(cudaErrorNotSupported);
}
cudaError_t cudaGraphCreate(cudaGraph_t *, unsigned) { return done(cudaErrorNotSupported); }
OK(cudaGraphDestroy, (cudaGraph_t))
OK(cudaGraphExecDestroy, (cudaGraphExec_t))
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return done(cudaErrorNotSupported); }
OK(cudaGraphLaunch, (cudaGraphExec_t, cudaStream_t))
}
