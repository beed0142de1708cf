// util.h -- error reporting shared by the host side of the library.
#pragma once
#include <cstddef>

#include "ps_b200.h"

// Records msg as the thread's last error and returns code.
ps_status psb_fail(ps_status code, const char *msg);
// Records a CUDA error (with the failing call's name) and returns PS_ERR_CUDA.
ps_status psb_fail_cuda(int cuda_error, const char *what);

// Device buffers from the library's own stream-ordered pool of the current
// device (pool.cu); alloc returns a cudaError_t value.
int psb_pool_alloc(int device, void **ptr, size_t bytes, void *stream);
void psb_pool_free(void *ptr, void *stream);
