// tce_pool.cu -- the pool of tce_pool.h.
#include "tce_pool.h"

#include <algorithm>
#include <mutex>

namespace tcehost {
namespace {

std::mutex g_mu;
long long g_handles = 0;
constexpr int MAX_DEV = 64;
cudaMemPool_t g_pool[MAX_DEV] = {};

// the current device's pool, made on first use; null when it cannot be made
cudaMemPool_t pool(bool make)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEV) return nullptr;
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_pool[dev] && make) {
        cudaMemPoolProps pr = {};
        pr.allocType = cudaMemAllocationTypePinned;
        pr.location.type = cudaMemLocationTypeDevice;
        pr.location.id = dev;
        unsigned long long keep = TCE_POOL_KEEP;
        if (cudaMemPoolCreate(&g_pool[dev], &pr) != cudaSuccess) {
            cudaGetLastError();
            g_pool[dev] = nullptr;
        } else {
            cudaMemPoolSetAttribute(g_pool[dev], cudaMemPoolAttrReleaseThreshold, &keep);
        }
    }
    return g_pool[dev];
}

bool no_handles()
{
    std::lock_guard<std::mutex> lock(g_mu);
    return g_handles == 0;
}

}  // namespace

PoolUser::PoolUser()
{
    std::lock_guard<std::mutex> lock(g_mu);
    ++g_handles;
}

PoolUser::~PoolUser()
{
    std::lock_guard<std::mutex> lock(g_mu);
    if (--g_handles > 0) return;
    int dev = 0;
    const bool have = cudaGetDevice(&dev) == cudaSuccess;
    for (int d = 0; d < MAX_DEV; ++d)
        if (g_pool[d] && cudaSetDevice(d) == cudaSuccess) {
            cudaDeviceSynchronize();   // frees still ordered behind running work
            cudaMemPoolTrimTo(g_pool[d], 0);
        }
    if (have) cudaSetDevice(dev);
}

bool pool_trim()
{
    cudaMemPool_t p = pool(false);
    if (!p) return false;
    cudaDeviceSynchronize();   // frees still ordered behind running work
    cudaMemPoolTrimTo(p, 0);
    return true;
}

cudaError_t device_malloc(void **p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        if (pool_trim()) e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
    }
    return e;
}

void *CallMemory::take(size_t bytes)
{
    Buffer b{nullptr, pooled_ + bytes <= TCE_POOL_KEEP && !no_handles()};
    cudaMemPool_t pl = b.pooled ? pool(true) : nullptr;
    cudaError_t e = cudaErrorMemoryAllocation;
    if (pl) {
        e = cudaMallocFromPoolAsync(&b.p, bytes, pl, st_);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            pool_trim();
            e = cudaMallocFromPoolAsync(&b.p, bytes, pl, st_);
        }
        if (e != cudaSuccess) cudaGetLastError();
    } else {
        b.pooled = false;
        e = device_malloc(&b.p, bytes);
    }
    if (e != cudaSuccess) return nullptr;
    if (b.pooled) pooled_ += bytes;
    mem_.push_back(b);
    return b.p;
}

// (cudaFree waits for the device's running work)
void CallMemory::give(const Buffer &b)
{
    if (b.pooled) cudaFreeAsync(b.p, st_);
    else cudaFree(b.p);
}

void CallMemory::drop(void *p)
{
    const auto it = std::find_if(mem_.begin(), mem_.end(), [&](const Buffer &b) { return b.p == p; });
    if (it == mem_.end()) return;
    give(*it);
    mem_.erase(it);
}

void CallMemory::drop_all()
{
    for (const Buffer &b : mem_) give(b);
    mem_.clear();
    pooled_ = 0;
}

CallMemory::~CallMemory() { drop_all(); }

}  // namespace tcehost
