// Test-only, included before mpmg_api.cu: its allocations can be made to fail
// (mpmg_test_fail_*), as on a device or a host without memory left.
#include <cuda_runtime.h>

extern "C" {
__attribute__((visibility("default"))) int mpmg_test_fail_device = -1;   // fail the device allocation this many calls on
__attribute__((visibility("default"))) int mpmg_test_fail_pinned = 0;    // fail every pinned allocation
}

static inline cudaError_t test_malloc(void **p, size_t n)
{
    if (mpmg_test_fail_device >= 0 && mpmg_test_fail_device-- == 0) return cudaErrorMemoryAllocation;
    return cudaMalloc(p, n);
}
static inline cudaError_t test_malloc_host(void **p, size_t n)
{
    return mpmg_test_fail_pinned ? cudaErrorMemoryAllocation : cudaMallocHost(p, n);
}
#define cudaMalloc(p, n) test_malloc((void **)(p), n)
#define cudaMallocHost(p, n) test_malloc_host((void **)(p), n)
