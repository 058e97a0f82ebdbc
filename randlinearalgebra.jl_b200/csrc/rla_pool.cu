// rla_pool.cu -- memory of objects that outlive a call: a bounded device pool shared by the
// contexts of a device, and pinned status slots.
#include <map>
#include <mutex>
#include <set>

#include "rla_internal.cuh"

namespace rla {

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    int contexts = 0;
};
static std::mutex g_pool_mu;
static std::map<int, DevicePool> &g_pool = *new std::map<int, DevicePool>;  // by device; lives as long as the process
// Buffers that the pool would not keep are mapped and unmapped by each allocation, which takes longer
// there: a Gaussian sketch created and destroyed, pool / cudaMalloc, 336 MB 0.64 / 1.05 ms, 400 MB 1.31 /
// 1.37, 666 MB 2.8 / 1.5, 1680 MB 9.5 / 2.9.
constexpr size_t POOL_MAX_ALLOC = 384ull << 20;
static std::set<void *> &g_large = *new std::set<void *>;  // from cudaMalloc

cudaError_t dev_alloc(rla_ctx *ctx, void **p, size_t bytes) {
    bytes = std::max<size_t>(bytes, 16);
    // an allocation that became part of a captured graph would be mapped only while the graph runs
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    const cudaError_t ec = cudaStreamIsCapturing(ctx->stream, &cap);
    if (ec != cudaSuccess) return ec;
    if (cap != cudaStreamCaptureStatusNone) return cudaErrorStreamCaptureUnsupported;
    if (bytes > POOL_MAX_ALLOC) {
        const cudaError_t e = cudaMalloc(p, bytes);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(g_pool_mu);
        g_large.insert(*p);
        return e;
    }
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_pool_mu);
        DevicePool &d = g_pool[ctx->device];
        if (!d.pool) {
            cudaMemPoolProps pp = {};
            pp.allocType = cudaMemAllocationTypePinned;
            pp.location.type = cudaMemLocationTypeDevice;
            pp.location.id = ctx->device;
            uint64_t keep = 256ull << 20;
            const cudaError_t e = cudaMemPoolCreate(&d.pool, &pp);
            if (e != cudaSuccess) {  // no other allocator: dev_free takes the rest for pool memory
                d.pool = nullptr;
                return e;
            }
            cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
        pool = d.pool;
    }
    return cudaMallocFromPoolAsync(p, bytes, pool, ctx->stream);
}

void dev_free(void *p, cudaStream_t stream) {
    if (!p) return;
    {
        std::unique_lock<std::mutex> lock(g_pool_mu);
        if (g_large.erase(p)) {
            lock.unlock();
            cudaFree(p);  // waits for the device
            return;
        }
    }
    cudaFreeAsync(p, stream);
}

static std::mutex g_slot_mu;
static char *g_slots = nullptr;
static uint64_t g_slots_used = 0;

cudaError_t pinned_slot(double **p) {
    std::lock_guard<std::mutex> lock(g_slot_mu);
    if (!g_slots) {
        const cudaError_t e = cudaHostAlloc((void **)&g_slots, 64 * 64, cudaHostAllocPortable);
        if (e != cudaSuccess) {
            g_slots = nullptr;
            return e;
        }
    }
    for (int i = 0; i < 64; ++i)
        if (!((g_slots_used >> i) & 1u)) {
            g_slots_used |= 1ull << i;
            *p = (double *)(g_slots + 64 * i);
            return cudaSuccess;
        }
    return cudaHostAlloc((void **)p, 64, cudaHostAllocPortable);
}

void pinned_slot_free(double *p) {
    if (!p) return;
    std::lock_guard<std::mutex> lock(g_slot_mu);
    const ptrdiff_t off = (char *)p - g_slots;
    if (g_slots && off >= 0 && off < 64 * 64) g_slots_used &= ~(1ull << (off / 64));
    else cudaFreeHost(p);
}

// The device's last context gives the pool's free memory back.
void pool_contexts(int device, int change) {
    std::lock_guard<std::mutex> lock(g_pool_mu);
    DevicePool &d = g_pool[device];
    d.contexts += change;
    if (d.contexts == 0 && d.pool) cudaMemPoolTrimTo(d.pool, 0);
}

}  // namespace rla
