#include "pool.h"

#include <map>
#include <mutex>
#include <vector>

namespace v2g {

namespace {

std::mutex g_mu;
// per device: the pool, or nullptr where the device has no stream-ordered allocator
std::map<int, cudaMemPool_t> g_pools;
std::multimap<size_t, void*> g_pinned;
size_t g_pinned_bytes = 0;
int g_owners = 0;

cudaMemPool_t pool_of(int device) {
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_pools.find(device);
    if (it != g_pools.end()) return it->second;
    cudaMemPool_t pool = nullptr;
    int ok = 0;
    if (cudaDeviceGetAttribute(&ok, cudaDevAttrMemoryPoolsSupported, device) == cudaSuccess && ok) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        unsigned long long keep = kPoolKeep;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            pool = nullptr;
        } else if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            pool = nullptr;
        }
        if (!pool) cudaGetLastError();
    }
    return g_pools[device] = pool;
}

size_t pinned_size(size_t bytes) {
    size_t s = 4096;
    while (s < bytes) s *= 2;
    return s;
}

}  // namespace

namespace {

// alloc(), once more without what the pool holds unused if that is in the way
template <class F>
cudaError_t retried(cudaMemPool_t pool, F&& alloc) {
    cudaError_t e = alloc();
    if (e == cudaErrorMemoryAllocation && pool) {
        cudaGetLastError();
        cudaStreamSynchronize(cudaStreamLegacy);
        cudaMemPoolTrimTo(pool, 0);
        e = alloc();
    }
    return e;
}

template <class F>
void on_device(int device, F&& f) {
    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != device) cudaSetDevice(device);
    f();
    if (prev >= 0 && prev != device) cudaSetDevice(prev);
}

}  // namespace

cudaError_t pool_alloc(void** p, size_t bytes) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const cudaMemPool_t pool = pool_of(device);
    if (!pool) return cudaMalloc(p, bytes);
    return retried(pool, [&] { return cudaMallocFromPoolAsync(p, bytes, pool, cudaStreamLegacy); });
}

void pool_free(void* p, int device) {
    if (!p) return;
    on_device(device, [&] {
        // refused where a caller's own capture forbids work on the legacy stream
        if (!pool_of(device) || cudaFreeAsync(p, cudaStreamLegacy) != cudaSuccess) cudaFree(p);
    });
}

cudaError_t device_alloc(void** p, size_t bytes) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    return retried(pool_of(device), [&] { return cudaMalloc(p, bytes); });
}

void device_free(void* p, int device) {
    if (!p) return;
    on_device(device, [&] { cudaFree(p); });
}

cudaError_t pinned_alloc(void** p, size_t bytes) {
    const size_t size = pinned_size(bytes);
    {
        std::lock_guard<std::mutex> lk(g_mu);
        auto it = g_pinned.find(size);
        if (it != g_pinned.end()) {
            *p = it->second;
            g_pinned.erase(it);
            g_pinned_bytes -= size;
            return cudaSuccess;
        }
    }
    return cudaMallocHost(p, size);
}

void pinned_free(void* p, size_t bytes) {
    if (!p) return;
    const size_t size = pinned_size(bytes);
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_pinned_bytes + size <= kPinnedKeep) {
            g_pinned.emplace(size, p);
            g_pinned_bytes += size;
            return;
        }
    }
    cudaFreeHost(p);
}

size_t pool_idle(int device) {
    const cudaMemPool_t pool = pool_of(device);
    unsigned long long reserved = 0, used = 0;
    if (!pool || cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess || used > reserved)
        return 0;
    return reserved - used;
}

PoolOwner::PoolOwner() {
    std::lock_guard<std::mutex> lk(g_mu);
    g_owners++;
}

PoolOwner::~PoolOwner() {
    std::map<int, cudaMemPool_t> pools;
    std::multimap<size_t, void*> pinned;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (--g_owners > 0) return;
        pools = g_pools;
        pinned.swap(g_pinned);
        g_pinned_bytes = 0;
    }
    for (const auto& b : pinned) cudaFreeHost(b.second);
    for (const auto& d : pools)
        if (d.second) on_device(d.first, [&] {
            cudaStreamSynchronize(cudaStreamLegacy);  // the frees queued there
            cudaMemPoolTrimTo(d.second, 0);
        });
}

}  // namespace v2g
