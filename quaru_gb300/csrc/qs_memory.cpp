// qs_memory.cpp — device memory kept between calls.
//
// Working buffers of a call (and small register states) come from a stream-ordered pool of the library's
// own instead of the device's default pool. The default pool gives every free byte back to CUDA
// at each synchronisation, so a call that allocates, works and waits pays for mapping its buffers anew:
// about 95 us of an 8-qubit gradient's 225 us. This pool keeps up to kKeepBytes free while the library has
// registers or batches, and one allocation unit once it has none; memory beyond that goes back as before,
// and all of it when an allocation fails.
#include <cuda_runtime.h>

#include <map>
#include <mutex>

#include "qs_kernels.h"

namespace qs {
namespace {

constexpr size_t kKeepBytes = size_t(64) << 20;
constexpr size_t kIdleBytes = size_t(2) << 20;

std::mutex g_mu;
std::map<int, cudaMemPool_t> g_pools;  // per device; null where a pool could not be had
int g_objects = 0;

cudaMemPool_t pool_of_current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lock(g_mu);
    const auto it = g_pools.find(dev);
    if (it != g_pools.end()) return it->second;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
        cudaGetLastError();
        pool = nullptr;
    } else {
        uint64_t keep = kKeepBytes;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    g_pools[dev] = pool;
    return pool;
}

void trim(size_t keep) {
    std::lock_guard<std::mutex> lock(g_mu);
    for (auto& p : g_pools)
        if (p.second) cudaMemPoolTrimTo(p.second, keep);
}

}  // namespace

cudaError_t device_alloc(void** p, size_t bytes, cudaStream_t s) {
    cudaMemPool_t pool = pool_of_current_device();
    auto get = [&] { return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s); };
    cudaError_t e = get();
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        give_back_memory();
        e = get();
    }
    return e;
}

void give_back_memory() { trim(0); }

void object_created() {
    std::lock_guard<std::mutex> lock(g_mu);
    g_objects++;
}

void object_destroyed() {
    bool last;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        last = --g_objects == 0;
    }
    if (last) trim(kIdleBytes);
}

}  // namespace qs
