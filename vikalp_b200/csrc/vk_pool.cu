// Memory pool of the library's solves (vk_common.cuh).
#include "vk_common.cuh"

#include <mutex>

namespace vk {
namespace {

constexpr int kMaxDevices = 64;

// The pool of the current device, made on first use; null when the device has
// no memory pools. Pools live until the process exits.
cudaMemPool_t device_pool() {
    static std::mutex mu;
    static cudaMemPool_t pools[kMaxDevices] = {};
    static bool tried[kMaxDevices] = {};
    int dev = 0;
    VK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (tried[dev]) return pools[dev];
    tried[dev] = true;
    int supported = 0;
    VK_CUDA(cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev));
    if (!supported) return nullptr;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    VK_CUDA(cudaMemPoolCreate(&pool, &props));
    unsigned long long keep = kPoolKeep;
    VK_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    return pools[dev] = pool;
}

} // namespace

void *pool_alloc(size_t bytes, cudaStream_t s) {
    void *p = nullptr;
    if (cudaMemPool_t pool = device_pool())
        VK_CUDA(cudaMallocFromPoolAsync(&p, bytes, pool, s));
    else
        VK_CUDA(cudaMalloc(&p, bytes));
    return p;
}

void pool_free(void *p, cudaStream_t s) noexcept {
    // cudaFree also takes pool memory; it waits for the device, as it must where
    // there are no pools
    if (cudaFreeAsync(p, s) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(p);
    }
}

} // namespace vk
