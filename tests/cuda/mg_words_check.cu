// Test-only kernels: the multigrid solve's conversions between FP32 and scaled
// FP64 (mg_wide, mg_narrow).  Built by tests/test_gpu_mg_words.py with nvcc into
// a temporary shared library.
#include "../../mpm-2d_gb300/csrc/mpmg_mg_words.cuh"

namespace {

__global__ void wide_kernel(long long n, const float *__restrict__ in, int e, double *__restrict__ out)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = mg_wide(in[i], e);
}

__global__ void narrow_kernel(long long n, const double *__restrict__ in, int e, float *__restrict__ out)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = mg_narrow(in[i], e);
}

}  // namespace

// in and out are device arrays of n entries.
extern "C" int widen(long long n, const float *in, int e, double *out)
{
    wide_kernel<<<256, 256>>>(n, in, e, out);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}

extern "C" int narrow(long long n, const double *in, int e, float *out)
{
    narrow_kernel<<<256, 256>>>(n, in, e, out);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
