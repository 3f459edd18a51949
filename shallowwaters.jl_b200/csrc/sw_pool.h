// sw_pool.h -- device blocks of the gradient, kept for reuse (sw_runtime.cu) in
// a pool of their own: bounded, keyed by size, device and CUDA context, the
// oldest going first, returned by sw_trim_memory.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace swb {

cudaError_t pool_malloc(void** p, size_t bytes);
// all work on the block must have ended
void pool_free(void* p, size_t bytes);

}  // namespace swb
