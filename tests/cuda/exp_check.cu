// Test-only: mat::exp_small of given arguments.  Built by tests/test_gpu_exp.py
// with nvcc into a temporary shared library.
#include "../../mpm-2d_gb300/csrc/mpmg_materials.cuh"

namespace {

__global__ void exp_kernel(int n, const double *x, double *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = mat::exp_small(x[i]);
}

}  // namespace

extern "C" int exp_of(int n, const double *x, double *out)
{
    double *d = nullptr;
    if (cudaMalloc(&d, 2 * (size_t)n * sizeof(double)) != cudaSuccess) return 1;
    int rc = cudaMemcpy(d, x, n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
    exp_kernel<<<(n + 127) / 128, 128>>>(n, d, d + n);
    rc |= cudaMemcpy(out, d + n, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    return rc;
}
