// fake_cudart.cc -- a CUDA runtime without a device, for CPU tests of the engine's
// host code: preloaded before libcudart, it keeps "device" memory in host memory,
// runs no kernel and writes one line per call of interest to $FAKE_CUDART_LOG.
#include <cuda_runtime_api.h>

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#undef cudaGetDeviceProperties
#define FAKE extern "C" __attribute__((visibility("default")))

namespace {

std::map<const void *, std::string> &names() {
    static std::map<const void *, std::string> m;
    return m;
}
std::map<const void *, void *> &symbols() {
    static std::map<const void *, void *> m;
    return m;
}
std::map<cudaEvent_t, unsigned> &event_flags() {
    static std::map<cudaEvent_t, unsigned> m;
    return m;
}
std::mutex mu;
struct {
    dim3 grid, block;
    size_t shared;
    cudaStream_t stream;
} config;
uintptr_t next_handle = 0x1000;

void say(const char *fmt, ...) {
    static FILE *f = [] {
        const char *path = std::getenv("FAKE_CUDART_LOG");
        return path ? std::fopen(path, "a") : stderr;
    }();
    std::lock_guard<std::mutex> g(mu);
    va_list ap;
    va_start(ap, fmt);
    std::vfprintf(f, fmt, ap);
    va_end(ap);
    std::fputc('\n', f);
    std::fflush(f);
}

template <typename T>
cudaError_t handle(T *out) {
    *out = reinterpret_cast<T>(next_handle += 16);
    return cudaSuccess;
}

void *symbol(const void *s) { return symbols().count(s) ? symbols()[s] : nullptr; }
const char *name(const void *s) { return names().count(s) ? names()[s].c_str() : "?"; }

}  // namespace

// registration
FAKE void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
FAKE void __cudaRegisterFatBinaryEnd(void **) {}
FAKE void __cudaUnregisterFatBinary(void **) {}
FAKE void __cudaRegisterFunction(void **, const char *host, char *, const char *device, int, uint3 *, uint3 *, dim3 *,
                                 dim3 *, int *) {
    names()[host] = device;
}
FAKE void __cudaRegisterVar(void **, char *host, char *, const char *device, int, size_t size, int, int) {
    names()[host] = device;
    symbols()[host] = std::calloc(1, size);
}
FAKE unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
    config = {grid, block, shared, stream};
    return 0;
}
FAKE cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *shared, void *stream) {
    *grid = config.grid;
    *block = config.block;
    *shared = config.shared;
    *(cudaStream_t *)stream = config.stream;
    return cudaSuccess;
}

// device
FAKE cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
FAKE cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
FAKE cudaError_t cudaSetDevice(int) { return cudaSuccess; }
FAKE cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
FAKE cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)180 << 30; return cudaSuccess; }
FAKE cudaError_t cudaGetLastError() { return cudaSuccess; }
FAKE const char *cudaGetErrorName(cudaError_t) { return "fake"; }
FAKE const char *cudaGetErrorString(cudaError_t) { return "fake"; }
FAKE cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *) { return cudaSuccess; }
FAKE cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
FAKE cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}

// memory
FAKE cudaError_t cudaMalloc(void **p, size_t n) {
    say("malloc %zu", n);
    *p = std::calloc(1, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) {
    *p = std::calloc(1, n);
    say("mallocasync %p %zu", *p, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaFree(void *p) {
    say("free %p", p);
    std::free(p);
    return cudaSuccess;
}
FAKE cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
    say("free %p", p);
    std::free(p);
    return cudaSuccess;
}
FAKE cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    say("hostalloc %zu", n);
    *p = std::calloc(1, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaFreeHost(void *p) {
    say("hostfree");
    std::free(p);
    return cudaSuccess;
}
FAKE cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
FAKE cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
FAKE cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
FAKE cudaError_t cudaMemcpyToSymbol(const void *s, const void *src, size_t n, size_t off, cudaMemcpyKind) {
    say("upload %s stream 0", name(s));
    std::memcpy((char *)symbol(s) + off, src, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaMemcpyToSymbolAsync(const void *s, const void *src, size_t n, size_t off, cudaMemcpyKind,
                                         cudaStream_t st) {
    say("upload %s stream %zx", name(s), (size_t)st);
    std::memcpy((char *)symbol(s) + off, src, n);
    return cudaSuccess;
}
FAKE cudaError_t cudaGetSymbolAddress(void **p, const void *s) { *p = symbol(s); return cudaSuccess; }

// streams, events, launches, graphs
FAKE cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle(s); }
FAKE cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    say("synchronize stream %zx", (size_t)s);
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    say("capture");
    return cudaSuccess;
}
FAKE cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return handle(g); }
FAKE cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
FAKE cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned flags) {
    const cudaError_t r = handle(e);
    event_flags()[*e] = flags;
    return r;
}
FAKE cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
FAKE cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    say("wait event %s", event_flags()[e] & cudaEventBlockingSync ? "blocking" : "spinning");
    return cudaSuccess;
}
FAKE cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t, cudaStream_t s) {
    say("launch %s stream %zx", name(f), (size_t)s);
    return cudaSuccess;
}
FAKE cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) {
    say("launch %s stream %zx", name(f), (size_t)c->stream);
    return cudaSuccess;
}
FAKE cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { return handle(e); }
FAKE cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
