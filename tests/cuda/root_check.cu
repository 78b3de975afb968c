// Test-only kernels: the library's FP64 square root, quotients
// (mat::root, mat::quot, mat::dvd_const) and product (mat::imul) against the IEEE
// operations, on random operands, on operands whose result lies next to a
// midpoint of two doubles or to a power of two, and on the ends of the range.
// Built by tests/test_gpu_root.py with nvcc into a temporary shared library.
#include <stdint.h>

#include "../../mpm-2d_gb300/csrc/mpmg_materials.cuh"

namespace {

__device__ uint64_t mix(uint64_t z)
{
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__device__ double bits(uint64_t b)
{
    return __longlong_as_double((long long)b);
}

// kind 0: any significand, exponents -span..span; 1: any bit pattern; 2: a
// significand within 8 ulps of a power of two; 3: a short significand.
__device__ double operand(uint64_t r, int kind, int span)
{
    const uint64_t frac = 0xfffffffffffffull;
    const uint64_t e = (uint64_t)(1023 - span + (int)((r >> 52) % (uint64_t)(2 * span + 1))) << 52;
    if (kind == 1) return bits(mix(r));
    if (kind == 2) return bits(e + ((r & 15) - 8));
    if (kind == 3) return bits(e | ((r & frac) & (frac << (20 + (r >> 40) % 32))));
    return bits(e | (r & frac));
}

enum { ROOT = 0, QUOT = 1, CONST = 2, MUL = 3 };

__global__ void check_kernel(int op, int kind, int span, mat::Known k, long long n, uint64_t seed,
                             unsigned long long *bad, double *example)
{
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const uint64_t r0 = mix(seed ^ (uint64_t)i), r1 = mix(r0);
        double a = operand(r0, kind & 3, span), b = operand(r1, (kind >> 2) & 3, span), got, want;
        const uint64_t half = 1ull << 28;   // FP32-exact heads: m (1 + 2^-53) needs 54 bits, so step from a double
        if (op == ROOT) {
            if (kind & 16) {
                // x next to the square of the midpoint above b
                b = fabs(b);
                const double u = bits((uint64_t)__double_as_longlong(b) + 1) - b;
                a = __fma_rn(b, u, __dmul_rn(b, b));
                a = bits((uint64_t)__double_as_longlong(a) + (r0 % 5) - 2);
            }
            a = (kind & 3) == 1 ? a : fabs(a);
            got = r1 & 2 ? mat::root(a) : mat::root<-1>(a);
            want = __dsqrt_rn(r1 & 2 ? a : 0.5 * a);
        } else if (op == QUOT) {
            if (kind & 16) {
                // a next to b times the midpoint above c
                const double c = operand(mix(r1 ^ half), 0, span);
                const double u = bits((uint64_t)__double_as_longlong(c) + 1) - c;
                a = __fma_rn(b, 0.5 * u, __dmul_rn(b, c));
                a = bits((uint64_t)__double_as_longlong(a) + (r0 % 5) - 2);
            }
            if (r1 & 1) b = -b;
            got = r1 & 2 ? mat::quot(a, b) : mat::quot<1>(a, b);
            want = __ddiv_rn(r1 & 2 ? a : 2.0 * a, b);
        } else if (op == MUL) {
            if (r1 & 1) b = -b;
            got = mat::imul(a, b);
            want = __dmul_rn(a, b);
        } else {
            if (kind & 16) {
                const double c = operand(mix(r1 ^ half), 0, span);
                const double u = bits((uint64_t)__double_as_longlong(c) + 1) - c;
                a = __fma_rn(k.b, 0.5 * u, __dmul_rn(k.b, c));
                a = bits((uint64_t)__double_as_longlong(a) + (r0 % 5) - 2);
            }
            got = mat::dvd_const(a, k);
            want = __ddiv_rn(a, k.b);
        }
        const bool same = __double_as_longlong(got) == __double_as_longlong(want) || (isnan(got) && isnan(want));
        if (!same && atomicAdd(bad, 1ull) == 0) {
            example[0] = a;
            example[1] = b;
            example[2] = got;
            example[3] = want;
        }
    }
}

}  // namespace

// Mismatches among n operands; kind: operand kind of a (bits 0-1) and b (bits
// 2-3), 16: results next to a midpoint.  b is the divisor of op 2.
extern "C" int check_op(int op, int kind, int span, double b, long long n, unsigned long long seed,
                        unsigned long long *mismatches, double *example)
{
    unsigned long long *d_bad = nullptr;
    double *d_ex = nullptr;
    if (cudaMalloc(&d_bad, sizeof(*d_bad)) != cudaSuccess) return 1;
    if (cudaMalloc(&d_ex, 4 * sizeof(double)) != cudaSuccess) return 1;
    cudaMemset(d_bad, 0, sizeof(*d_bad));
    cudaMemset(d_ex, 0, 4 * sizeof(double));
    const mat::Known k = mat::make_known(b);
    check_kernel<<<1216, 256>>>(op, kind, span, k, n, seed, d_bad, d_ex);
    cudaError_t e = cudaMemcpy(mismatches, d_bad, sizeof(*d_bad), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(example, d_ex, 4 * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(d_bad);
    cudaFree(d_ex);
    return e == cudaSuccess ? 0 : 1;
}
