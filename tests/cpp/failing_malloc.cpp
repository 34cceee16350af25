// cudaMalloc as the library sees it in tests/test_gpu_batch_memory.py: the
// objects of the build are linked again with --wrap=cudaMalloc, so that requests
// above a limit are refused on the host with the runtime's own error code and
// the GPU's memory is never exhausted.
#include <cuda_runtime_api.h>

#include <cstddef>

static size_t limit_bytes = ~(size_t)0;
static int refused = 0;

extern "C" __attribute__((visibility("default"))) void malloc_limit(size_t bytes) {
    limit_bytes = bytes;
    refused = 0;
}
extern "C" __attribute__((visibility("default"))) int malloc_refused(void) { return refused; }

extern "C" cudaError_t __real_cudaMalloc(void **p, size_t bytes);
extern "C" cudaError_t __wrap_cudaMalloc(void **p, size_t bytes) {
    if (bytes > limit_bytes) {
        refused++;
        return cudaErrorMemoryAllocation;
    }
    return __real_cudaMalloc(p, bytes);
}
