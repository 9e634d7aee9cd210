// memory.cu -- device memory for problems and engines: a stream-ordered pool per device,
// owned by the library.  Freed blocks stay cached in the pool (release threshold = max),
// so creating and destroying engines at serving rates costs no device-wide
// synchronisation and no page mapping after the first time.
#include <cstdint>
#include <map>
#include <mutex>
#include <vector>

#include "engine.h"

namespace bk {

static std::mutex g_pool_mu;
static std::map<int, cudaMemPool_t> g_pools;

static cudaError_t pool_of(int dev, cudaMemPool_t* out) {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pools.find(dev);
    if (it != g_pools.end()) {
        *out = it->second;
        return cudaSuccess;
    }
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool;
    cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = UINT64_MAX;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) return e;
    g_pools[dev] = pool;
    *out = pool;
    return cudaSuccess;
}

int32_t dev_alloc(void** p, size_t bytes, cudaStream_t st) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    cudaMemPool_t pool;
    if (e == cudaSuccess) e = pool_of(dev, &pool);
    if (e != cudaSuccess) return cuda_fail(e, "memory pool");
    e = cudaMallocFromPoolAsync(p, bytes ? bytes : 16, pool, st);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(BRKGA_ERR_OOM, std::string("device allocation of ") + std::to_string(bytes) + " bytes: " +
                                       cudaGetErrorString(e));
    }
    return BRKGA_OK;
}

void dev_free(void* p, cudaStream_t st) {
    if (p) cudaFreeAsync(p, st);
}

// bytes the pool holds but has not handed out (reusable without a new device allocation)
size_t pool_spare(int dev) {
    cudaMemPool_t pool;
    if (pool_of(dev, &pool) != cudaSuccess) return 0;
    uint64_t reserved = 0, used = 0;
    cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved);
    cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used);
    return reserved > used ? (size_t)(reserved - used) : 0;
}

size_t pool_reserved(int dev) {
    cudaMemPool_t pool;
    if (pool_of(dev, &pool) != cudaSuccess) return 0;
    uint64_t v = 0;
    cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &v);
    return (size_t)v;
}

// Pinned words that kernels write when a wait between their CTAs runs out, so that a call which
// waits for its stream anyway sees it without a copy.  Handed out of pages of 1024 (allocating
// one costs tens of microseconds); a page that is not in use is given back unless it is the last.
struct FlagPage {
    int32_t* base;
    std::vector<int32_t*> spare;
};
constexpr int kFlagsPerPage = 1024;
static std::mutex g_flag_mu;
static std::vector<FlagPage> g_flag_pages;

int32_t flag_take(int32_t** out) {
    std::lock_guard<std::mutex> lk(g_flag_mu);
    FlagPage* from = nullptr;
    for (FlagPage& p : g_flag_pages)
        if (!p.spare.empty()) from = &p;
    if (!from) {
        FlagPage p{};
        const cudaError_t e = cudaHostAlloc(&p.base, kFlagsPerPage * sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return fail(BRKGA_ERR_OOM, std::string("pinned flags: ") + cudaGetErrorString(e));
        }
        for (int i = kFlagsPerPage; i-- > 0;) p.spare.push_back(p.base + i);
        g_flag_pages.push_back(std::move(p));
        from = &g_flag_pages.back();
    }
    *out = from->spare.back();
    from->spare.pop_back();
    **out = 0;
    return BRKGA_OK;
}

void flag_give(int32_t* f) {
    if (!f) return;
    std::lock_guard<std::mutex> lk(g_flag_mu);
    for (size_t i = 0; i < g_flag_pages.size(); ++i) {
        FlagPage& p = g_flag_pages[i];
        if (f < p.base || f >= p.base + kFlagsPerPage) continue;
        p.spare.push_back(f);
        if ((int)p.spare.size() == kFlagsPerPage && g_flag_pages.size() > 1) {
            cudaFreeHost(p.base);
            g_flag_pages.erase(g_flag_pages.begin() + (long)i);
        }
        return;
    }
}

}  // namespace bk
