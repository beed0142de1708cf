// pool.cu -- short-lived device buffers of the screening entry points.
//
// cudaMalloc and cudaFree cost more than those calls' kernels, so buffers come
// from a stream-ordered pool of the library's own, one per device.  It keeps
// at most kKept bytes between calls; what it keeps unused the driver takes
// back when another allocation of the process runs short of memory.  A buffer
// is used and freed in the order of one stream, so threads and streams share
// the pool safely.
#include <cuda_runtime.h>

#include <mutex>

#include "util.h"

namespace {

constexpr int kMaxDevices = 64;
constexpr unsigned long long kKept = 32ull << 20;

std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices];

cudaError_t pool_of(int device, cudaMemPool_t *pool)
{
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_pool[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t p = nullptr;
        cudaError_t e = cudaMemPoolCreate(&p, &props);
        if (e != cudaSuccess) return e;
        unsigned long long keep = kKept;
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

int psb_pool_alloc(int device, void **ptr, size_t bytes, void *stream)
{
    cudaMemPool_t pool = nullptr;
    cudaError_t e = pool_of(device, &pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(ptr, bytes, pool, (cudaStream_t)stream);
    return (int)e;
}

void psb_pool_free(void *ptr, void *stream)
{
    if (ptr) cudaFreeAsync(ptr, (cudaStream_t)stream);
}
