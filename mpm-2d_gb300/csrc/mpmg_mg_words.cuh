// Conversions between the FP64 outer iteration of the multigrid solve and its
// FP32 V-cycle.
#pragma once
#include <stdint.h>

// 2^e times an FP32 value (subnormals as zero) as a double, and 2^e times a
// double rounded to FP32 (below FP32's normal range: zero), in integer
// arithmetic: the conversion instructions run on the FP64 pipe.  Both are for
// vectors of order one and |e| < 800; infinities and NaN stay what they are, and
// what FP32 cannot hold becomes an infinity, so that an overflow in the V-cycle
// ends the solve instead of passing for a number.
__device__ __forceinline__ double mg_wide(float f, int e)
{
    const unsigned b = __float_as_uint(f), m = b & 0x7fffffffu;
    if (m < 0x00800000u) return 0.0;
    const unsigned up = m >= 0x7f800000u ? 1792u << 20 : (unsigned)(896 + e) << 20;
    return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + up)), (int)(b << 29));
}

__device__ __forceinline__ float mg_narrow(double x, int e)
{
    const long long b = __double_as_longlong(x);
    const unsigned long long m = (unsigned long long)b & 0x7fffffffffffffffULL;
    const int f = (int)(m >> 52) + e;       // exponent field, double's bias
    const unsigned sign = (unsigned)((unsigned long long)b >> 32 & 0x80000000u);
    if (f < 897) return 0.0f;
    if (f > 1150) return __uint_as_float(sign | (m > 0x7ff0000000000000ULL ? 0x7fc00000u : 0x7f800000u));
    const unsigned long long r = (m + 0x0fffffffULL + ((m >> 29) & 1)) >> 29;   // to nearest even
    return __uint_as_float(sign | ((unsigned)r + ((unsigned)(e - 896) << 23)));
}
