// The per-device scratch pools (dev_scratch.h).
#include "dev_scratch.h"

#include <cstdint>
#include <mutex>

namespace panns {
namespace {

constexpr int kMaxDevices = 64;
std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices] = {nullptr};

cudaError_t device_pool(int device, cudaMemPool_t *pool) {
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_pool[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t p = nullptr;
        cudaError_t e = cudaMemPoolCreate(&p, &props);
        if (e != cudaSuccess) return e;
        uint64_t keep = kScratchKeep;
        e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(p);
            return e;
        }
        g_pool[device] = p;
    }
    *pool = g_pool[device];
    return cudaSuccess;
}

}  // namespace

cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    cudaMemPool_t pool = nullptr;
    if (e == cudaSuccess) e = device_pool(device, &pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(p, bytes, pool, s);
    return e;
}

void scratch_free(void *p, cudaStream_t s) { cudaFreeAsync(p, s); }

void scratch_trim(int device) {
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (device >= 0 && device < kMaxDevices) pool = g_pool[device];
    }
    if (pool) cudaMemPoolTrimTo(pool, 0);
}

cudaError_t allow_shared(const void *kern) {
    cudaFuncAttributes a{};
    const cudaError_t e = cudaFuncGetAttributes(&a, kern);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int) ((227u << 10) - a.sharedSizeBytes));
}

}  // namespace panns
