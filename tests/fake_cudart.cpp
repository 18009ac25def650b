// A stand-in for the CUDA runtime on a machine without a GPU: loaded before
// libtroy_b200.so (same soname), it runs the library's host code and records what it asks
// of the device. Device memory is host memory, kernels do nothing.
//
// A host-to-device cudaMemcpy from pageable memory may return before the data is on the
// device, and only the legacy stream (and what is synchronised with it) is ordered after
// it. So each such copy, and each kernel on the legacy stream, is "pending" until that stream
// is synchronised, and a kernel launched on another stream meanwhile is reported as a race.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
std::mutex mu;
std::map<const void *, std::string> names;
std::string record;
size_t pending = 0;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local Config config;

void line(const char *fmt, unsigned long long a = 0, unsigned long long b = 0, unsigned long long c = 0,
          unsigned long long d = 0) {
    char buf[256];
    std::snprintf(buf, sizeof buf, fmt, a, b, c, d);
    record += buf;
    record += '\n';
}
bool legacy(cudaStream_t s) { return s == nullptr || s == cudaStreamLegacy; }
unsigned long long num(const void *p) { return (unsigned long long)(uintptr_t)p; }
template <class T>
cudaError_t handle(T *out) {
    static uintptr_t next = 0x10000;
    std::lock_guard<std::mutex> g(mu);
    *out = reinterpret_cast<T>(next += 16);
    return cudaSuccess;
}
cudaError_t allocate(const char *how, void **p, size_t bytes) {
    *p = std::aligned_alloc(256, (bytes + 255) / 256 * 256 + 256);
    if (!*p) return cudaErrorMemoryAllocation;
    std::lock_guard<std::mutex> g(mu);
    record += how;
    line(" %llu %llu", num(*p), bytes);
    return cudaSuccess;
}
}  // namespace

extern "C" {
// ---- for the tests
void fake_reset() {
    std::lock_guard<std::mutex> g(mu);
    record.clear();
}
const char *fake_record() { return record.c_str(); }

// ---- registration and launches
void **__cudaRegisterFatBinary(void *) {
    static void *h = nullptr;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *device, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    names[host] = device;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    config = Config{grid, block, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *static_cast<cudaStream_t *>(s) = config.stream;
    return cudaSuccess;
}
// "launch <stream> <blocks> <threads> <first two words of the first argument> <name>": the
// words only for transforms, whose first argument starts with its input and output.
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3 block, void **args, size_t, cudaStream_t s) {
    std::lock_guard<std::mutex> g(mu);
    const std::string &name = names[f];
    if (legacy(s)) pending++;
    else if (pending) record += "race " + name + "\n";
    unsigned long long w[2] = {0, 0};
    if (name.find("Op") != std::string::npos) std::memcpy(w, args[0], sizeof w);
    char head[160];
    std::snprintf(head, sizeof head, "launch %llu %llu %u %llu %llu ", num(s), 1ull * grid.x * grid.y * grid.z,
                  block.x * block.y * block.z, w[0], w[1]);
    record += head + name + "\n";
    return cudaSuccess;
}

// ---- memory
cudaError_t cudaMalloc(void **p, size_t n) { return allocate("malloc", p, n); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return allocate("malloc_async", p, n); }
cudaError_t cudaFree(void *p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, cudaMemcpyKind kind) {
    std::memcpy(dst, src, n);
    std::lock_guard<std::mutex> g(mu);
    pending += kind == cudaMemcpyHostToDevice;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    std::lock_guard<std::mutex> g(mu);
    line("copy %llu %llu %llu %llu", num(s), num(dst), num(src), n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *dst, size_t, const void *src, size_t, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t s) {
    std::lock_guard<std::mutex> g(mu);
    line("copy %llu %llu %llu %llu", num(s), num(dst), num(src), w * h);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return allocate("symbol", p, 16); }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *pool, int) { return handle(pool); }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::mutex> g(mu);
    if (legacy(s)) pending = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *c) {
    *c = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { return handle(e); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}

// ---- device
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
    *n = 16;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
}
