// A host-only stand-in for the CUDA runtime: memory is host memory, launches are recorded by
// kernel name and not run, and every call that allocates, frees, copies, launches or waits is
// written to a log in order.  Linked with the library's own objects (fake_cuda.py) it lets tests
// check, without a GPU, which kernels a call launches and in which order buffers are used and
// released, and make a chosen call fail.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {
std::recursive_mutex mu;
std::string log_text;
// registered by the static constructors of the library's objects, before this file's own
std::map<const void *, std::string> &kernels() {
    static std::map<const void *, std::string> k;
    return k;
}
std::map<std::string, int> fail_after;  // call name -> calls that still succeed
bool capturing = false;
cudaError_t last = cudaSuccess;
uintptr_t handles = 0x1000;

void note(const char *fmt, ...) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    char buf[2048];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    log_text += buf;
    log_text += '\n';
}
cudaError_t set(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
bool failing(const char *call) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    auto it = fail_after.find(call);
    if (it == fail_after.end()) return false;
    return it->second-- <= 0;
}
template <class H>
cudaError_t handle(H *out) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    *out = reinterpret_cast<H>(handles += 16);
    return cudaSuccess;
}
cudaError_t allocate(const char *call, void **p, size_t bytes, const void *stream) {
    if (failing(call)) {
        *p = nullptr;
        return set(cudaErrorMemoryAllocation);
    }
    void *q = nullptr;  // aligned as device memory is; calloc keeps large buffers untouched
    q = calloc(1, bytes + 256 + sizeof(void *));
    *p = reinterpret_cast<void *>((reinterpret_cast<uintptr_t>(q) + 255) / 256 * 256);
    note("%s %p stream=%p", call, *p, stream);
    return cudaSuccess;
}
CUresult encode_tiled(...) { return CUDA_SUCCESS; }
}  // namespace

extern "C" {

// ---- for the tests ----
const char *fake_log(void) { return log_text.c_str(); }
void fake_reset(void) {
    std::lock_guard<std::recursive_mutex> lock(mu);
    log_text.clear();
    fail_after.clear();
    capturing = false;
    last = cudaSuccess;
}
void fake_fail_after(const char *call, int ok) { fail_after[call] = ok; }
void fake_capturing(int on) { capturing = on != 0; }

// ---- registration and launches ----
void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *) {
    kernels()[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
static thread_local struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} cfg;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *stream) {
    cfg = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = cfg.grid;
    *block = cfg.block;
    *smem = cfg.smem;
    *static_cast<cudaStream_t *>(stream) = cfg.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t smem, cudaStream_t s) {
    if (failing("launch")) return set(cudaErrorLaunchFailure);
    note("launch %s grid=%u,%u,%u block=%u smem=%zu stream=%p", kernels()[f].c_str(), g.x, g.y, g.z, b.x * b.y * b.z, smem, (void *)s);
    return cudaSuccess;
}

// ---- memory ----
cudaError_t cudaMalloc(void **p, size_t n) { return allocate("cudaMalloc", p, n, nullptr); }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t s) { return allocate("cudaMallocAsync", p, n, s); }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t s) {
    return allocate("cudaMallocFromPoolAsync", p, n, s);
}
cudaError_t cudaFree(void *p) {
    note("cudaFree %p", p);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t s) {
    note("cudaFreeAsync %p stream=%p", p, (void *)s);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return allocate("cudaHostAlloc", p, n, nullptr); }
cudaError_t cudaFreeHost(void *p) {
    note("cudaFreeHost %p", p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    note("cudaMemcpy %p", d);
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    note("cudaMemcpyAsync %p stream=%p bytes=%zu", d, (void *)st, n);
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
    if (failing("cudaMemsetAsync")) return set(cudaErrorUnknown);
    note("cudaMemsetAsync %p stream=%p", d, (void *)st);
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) {
    if (failing("cudaMemPoolCreate")) return set(cudaErrorNotSupported);
    return handle(p);
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) {
    note("cudaMemPoolTrimTo");
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) {
    *p = const_cast<void *>(sym);
    return cudaSuccess;
}

// ---- streams and events ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    if (failing("cudaStreamCreateWithFlags")) return set(cudaErrorUnknown);
    return handle(s);
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    note("cudaStreamSynchronize stream=%p", (void *)s);
    return capturing ? set(cudaErrorStreamCaptureUnsupported) : cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) {
    note("cudaDeviceSynchronize");
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
    *st = capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    if (failing("cudaEventCreateWithFlags")) return set(cudaErrorUnknown);
    return handle(e);
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }

// ---- device ----
cudaError_t cudaGetDeviceCount(int *n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMultiProcessorCount ? 148 : 232448;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    memset(a, 0, sizeof *a);
    a->ptxVersion = a->binaryVersion = 100;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *, void **fn, unsigned long long, cudaDriverEntryPointQueryResult *r) {
    *fn = reinterpret_cast<void *>(&encode_tiled);
    if (r) *r = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError(void) { return last; }
const char *cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }

}  // extern "C"
