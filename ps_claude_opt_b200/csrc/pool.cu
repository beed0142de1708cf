// pool.cu -- short-lived device buffers of the screening features.
//
// cudaMalloc and cudaFree cost more than that call's kernel, so its buffer comes
// from a stream-ordered pool of the library's own, one per device.  It keeps
// at most kKept bytes between calls; what it keeps unused the driver takes
// back when another allocation of the process runs short of memory.  A buffer
// is used and freed in the order of one stream, so threads and streams share
// the pool safely.  A pool belongs to the context it was made in: after a
// cudaDeviceReset the device has another context, and gets another pool.
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>

#include "util.h"

namespace {

constexpr int kMaxDevices = 64;
constexpr unsigned long long kKept = 32ull << 20;

struct Pool {
    cudaMemPool_t pool = nullptr;
    unsigned long long context = 0;
};

std::mutex g_mu;
Pool g_pool[kMaxDevices];

// Id of the current device's context: no two contexts of a process have the
// same, unlike their addresses.
cudaError_t context_id(unsigned long long *id)
{
    using Fn = CUresult (*)(CUcontext, unsigned long long *);
    static const Fn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (Fn)p;
    }();
    return fn && fn(nullptr, id) == CUDA_SUCCESS ? cudaSuccess : cudaErrorDeviceUninitialized;
}

// The current device's pool.
cudaError_t pool_of(int device, cudaMemPool_t *pool)
{
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    unsigned long long context = 0;
    const cudaError_t ce = context_id(&context);
    if (ce != cudaSuccess) return ce;
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_pool[device].context != context) {  // none yet, or of a context that is gone
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
        g_pool[device] = {p, context};
    }
    *pool = g_pool[device].pool;
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
