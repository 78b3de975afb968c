// Test-only kernels: the multigrid solve's conversions between FP32 and scaled
// FP64 (mg_wide, mg_narrow) and its bounded waits (mg_stage, mg_gather4), run by
// one block that plays block 0 of `nblocks` while the host has written the other
// blocks' words, or not.  Built by tests/test_gpu_mg_words.py with nvcc into a
// temporary shared library, with a low poll limit.
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

// out: the four totals, then 1 where the gather answered true.  stage: first
// stage nn words and store them, so that a wait that runs out precedes the
// gather.
__global__ void __launch_bounds__(kMgThreads) wait_kernel(unsigned long long *words, int nblocks,
                                                          const unsigned long long *staged, int nn, float *floats,
                                                          unsigned tag, int *status, double *out)
{
    __shared__ double scratch[4 * kMgThreads + 4];
    __shared__ float d0[64];
    if (threadIdx.x == 0) mg_gave_up() = 0;
    __syncthreads();
    if (nn > 0) {
        mg_stage(staged, nn, 0, nn, d0, 0, 0, d0, tag, status);
        for (int k = threadIdx.x; k < nn; k += blockDim.x) floats[k] = d0[k];
    }
    double v[4] = {1.0, 2.0, 3.0, 4.0};
    const bool ok = mg_gather4(mat::Unit{1.0, -0.0}, words, v, nblocks, scratch, tag, status);
    if (threadIdx.x == 0) {
        for (int c = 0; c < 4; c++) out[c] = v[c];
        out[4] = ok ? 1.0 : 0.0;
    }
}

}  // namespace

// words, staged, floats, status and out are device arrays; nn <= 64.
extern "C" int wait_block(unsigned long long *words, int nblocks, const unsigned long long *staged, int nn,
                          float *floats, unsigned tag, int *status, double *out)
{
    wait_kernel<<<1, kMgThreads>>>(words, nblocks, staged, nn, floats, tag, status, out);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}

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
