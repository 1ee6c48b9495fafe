// lbm_memory.cu -- device memory of the handles: one stream-ordered CUDA memory
// pool per device, so that a program that makes one handle after another (an
// optimiser that evaluates a gradient per iteration) does not pay for mapping
// and unmapping the same memory each time.
//
// Measured on GB300: freeing a gradient evaluation's 50 GB at 256^3 took 39 ms
// and allocating them 8 ms of 166 ms; from the pool the two take 0.1 ms.  64^3
// (40 buffers): 2.9 of 6.3 ms.
//
// The pool is the library's own, not the device's default one.  It keeps at
// most a quarter of the device's memory once the handles are gone (its release
// threshold; what is beyond goes back at the next synchronisation), and what it
// keeps is still there for the rest of the process: an allocation that does
// not fit beside it makes the driver release it (measured: cudaMalloc of 266
// GB succeeds on a 296 GB device whose pool holds 50 GB).  Allocations and
// frees are ordered on the handle's stream; the driver orders a block's next
// user behind them, whatever its stream or thread.
#include <cstdint>
#include <map>
#include <mutex>

#include <cudaTypedefs.h>

#include "lbm_handle.h"

namespace {

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    unsigned long long context = 0;  // the context the pool was made in
};

std::mutex g_mu;
std::map<int, DevicePool> g_pools;

// Identity of the current context (0: unknown): a pool does not outlive a
// cudaDeviceReset, and its handle must not be used after one.
unsigned long long context_id()
{
    static PFN_cuCtxGetId_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuCtxGetId_v12000>(p);
    });
    unsigned long long id = 0;
    if (!fn || fn(nullptr, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// The pool of the current device (null: none, plain cudaMalloc then).
cudaMemPool_t device_pool(int device)
{
    const unsigned long long ctx = context_id();
    if (ctx == 0) return nullptr;
    std::lock_guard<std::mutex> lock(g_mu);
    DevicePool &d = g_pools[device];
    if (d.pool && d.context == ctx) return d.pool;
    d.pool = nullptr;
    int has = 0;
    size_t freeb = 0, total = 0;
    if (cudaDeviceGetAttribute(&has, cudaDevAttrMemoryPoolsSupported, device) != cudaSuccess || !has ||
        cudaMemGetInfo(&freeb, &total) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    cudaMemPoolProps p = {};
    p.allocType = cudaMemAllocationTypePinned;
    p.handleTypes = cudaMemHandleTypeNone;
    p.location.type = cudaMemLocationTypeDevice;
    p.location.id = device;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    uint64_t keep = total / 4;
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaGetLastError();
        cudaMemPoolDestroy(pool);
        return nullptr;
    }
    d.pool = pool;
    d.context = ctx;
    return pool;
}

}  // namespace

namespace lbm {

cudaError_t device_alloc(lbm_t *h, void **p, size_t bytes)
{
    if (!h->pool_looked_up) {
        h->pool = device_pool(h->cfg.device);
        h->pool_looked_up = true;
    }
    return h->pool ? cudaMallocFromPoolAsync(p, bytes, h->pool, h->stream) : cudaMalloc(p, bytes);
}

void device_free(lbm_t *h, void *p)
{
    if (!p) return;
    if (h->pool) cudaFreeAsync(p, h->stream);
    else cudaFree(p);
}

size_t device_cached(const lbm_t *h)
{
    uint64_t reserved = 0, used = 0;
    if (!h->pool || cudaMemPoolGetAttribute(h->pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(h->pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
        return 0;
    return reserved > used ? (size_t)(reserved - used) : 0;
}

}  // namespace lbm
