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
// threshold), and a block that would take it beyond that is a cudaMalloc of its
// own: the pool maps new memory at 1.0 ms per GB and would unmap it at 0.7 on
// every such use (cudaMalloc 0.03, cudaFree 0.33), and its blocks of 80 GB and
// more are read slower.  256^3 backward sweeps, total ms from handle to handle,
// FP16 T = 2000 with 250 GB: all from the pool 1912, with this rule 1539, all from
// cudaMalloc 1645; FP32 T = 400 with 110 GB: 414, 355, 406.  What the pool
// keeps is there for the rest of the process: an allocation that does not fit
// beside it makes the driver release it (measured: cudaMalloc of 266 GB succeeds
// on a 296 GB device whose pool holds 50 GB), but another process cannot have
// it.  lbm_keep_memory sets how much that is, down to nothing (every block a
// cudaMalloc then), and gives what is idle beyond it back.  Allocations and
// frees are ordered on the handle's stream; the driver orders a block's next
// user behind them, whatever its stream or thread.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>

#include <cudaTypedefs.h>

#include "lbm_handle.h"

namespace {

struct DevicePool {
    cudaMemPool_t pool = nullptr;
    unsigned long long context = 0;  // the context the pool was made in
    size_t keep = 0;                 // bytes it keeps when unused
    size_t plain = 0;                // bytes of the handles' blocks beside it
    bool chosen = false;             // keep was set by lbm_keep_memory
};

std::mutex g_mu;
std::map<int, DevicePool> g_pools;

constexpr size_t kDefaultKeep = (size_t)-1;  // a quarter of the device's memory

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
    d.plain = 0;
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
    uint64_t keep = d.chosen ? d.keep : total / 4;
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaGetLastError();
        cudaMemPoolDestroy(pool);
        return nullptr;
    }
    d.pool = pool;
    d.context = ctx;
    d.keep = (size_t)keep;
    return pool;
}

size_t pool_keep(int device)
{
    std::lock_guard<std::mutex> lock(g_mu);
    return g_pools[device].keep;
}

size_t pool_used(cudaMemPool_t pool)
{
    uint64_t used = 0;
    return cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess ? (size_t)used : 0;
}

}  // namespace

namespace lbm {

bool page_locked(const void *p, size_t bytes)
{
    for (const char *at : {static_cast<const char *>(p), static_cast<const char *>(p) + bytes - 1}) {
        cudaPointerAttributes pa;
        if (cudaPointerGetAttributes(&pa, at) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (pa.type != cudaMemoryTypeHost) return false;
    }
    return true;
}

void make_pages(void *host, size_t bytes)
{
#ifdef MADV_POPULATE_WRITE
    // only a hint: the copies meet whatever pages it leaves
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), p = (uintptr_t)host;
    const uintptr_t first = (p + page - 1) / page * page, last = (p + bytes) / page * page;
    if (last > first) madvise((void *)first, last - first, MADV_POPULATE_WRITE);
#endif
}

cudaError_t device_alloc(lbm_t *h, void **p, size_t bytes)
{
    if (!h->pool_looked_up) {
        h->pool = device_pool(h->cfg.device);
        h->pool_looked_up = true;
    }
    if (!h->pool) return cudaMalloc(p, bytes);
    if (pool_used(h->pool) + bytes > pool_keep(h->cfg.device)) {
        const cudaError_t e = cudaMalloc(p, bytes);
        if (e == cudaSuccess) {
            h->plain.emplace_back(*p, bytes);
            std::lock_guard<std::mutex> lock(g_mu);
            g_pools[h->cfg.device].plain += bytes;
        }
        if (e != cudaErrorMemoryAllocation) return e;
        cudaGetLastError();  // perhaps beside blocks whose frees are still queued: the pool waits for those
    }
    return cudaMallocFromPoolAsync(p, bytes, h->pool, h->stream);
}

void device_free(lbm_t *h, void *p)
{
    if (!p) return;
    const auto own = std::find_if(h->plain.begin(), h->plain.end(), [p](const auto &b) { return b.first == p; });
    if (own != h->plain.end()) {
        std::lock_guard<std::mutex> lock(g_mu);
        g_pools[h->cfg.device].plain -= own->second;
        h->plain.erase(own);
    } else if (h->pool) {
        cudaFreeAsync(p, h->stream);
        return;
    }
    cudaFree(p);
}

size_t device_cached(const lbm_t *h)
{
    uint64_t reserved = 0;
    if (!h->pool || cudaMemPoolGetAttribute(h->pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess)
        return 0;
    const size_t used = pool_used(h->pool);
    return reserved > used ? (size_t)reserved - used : 0;
}

size_t device_in_use(const lbm_t *h)
{
    if (!h->pool) return h->base_bytes + h->adj.bytes;
    std::lock_guard<std::mutex> lock(g_mu);
    return pool_used(h->pool) + g_pools[h->cfg.device].plain;
}

cudaError_t keep_memory(int device, size_t bytes)
{
    const DeviceScope dev(device);
    std::lock_guard<std::mutex> lock(g_mu);
    DevicePool &d = g_pools[device];
    d.chosen = bytes != kDefaultKeep;
    if (d.chosen) d.keep = bytes;
    if (!d.pool) return cudaSuccess;  // it will be made with that
    cudaSetDevice(device);            // a thread of its own may have no context yet
    if (d.context != context_id()) return cudaSuccess;
    uint64_t keep = bytes;
    if (!d.chosen) {
        size_t freeb = 0, total = 0;
        const cudaError_t e = cudaMemGetInfo(&freeb, &total);
        if (e != cudaSuccess) return e;
        keep = d.keep = total / 4;
    }
    const cudaError_t e = cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
    return e == cudaSuccess ? cudaMemPoolTrimTo(d.pool, (size_t)keep) : e;
}

}  // namespace lbm
