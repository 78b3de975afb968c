// What the blocks of the multigrid solve pass to each other: tagged words and
// the waits for them, and the conversions between the FP64 outer iteration and
// the FP32 V-cycle.
#pragma once
#include <stdint.h>

#include "mpmg_internal.cuh"
#include "mpmg_materials.cuh"

constexpr int kMgThreads = 512;
constexpr int kMgBlocks = 160;         // blocks of the solve at most (mg_gather4: five a lane)
// polls of one wait before it gives up (a poll is one L2 round trip, about
// a microsecond: a few seconds in all); a build may set it lower to see a wait
// run out
#ifndef MPMG_MG_POLL_LIMIT
#define MPMG_MG_POLL_LIMIT (1ll << 22)
#endif
constexpr long long kMgPollLimit = MPMG_MG_POLL_LIMIT;
// sleep of a waiting warp between its rounds of loads (ns)
constexpr unsigned kMgNap = 40;

__device__ __forceinline__ unsigned long long mg_ld(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}

__device__ __forceinline__ void mg_st(unsigned long long *p, float x, unsigned tag)
{
    const unsigned long long v = ((unsigned long long)tag << 32) | (unsigned long long)__float_as_uint(x);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v));
}

// A word that needs no wait: value 0 with the current tag.
__device__ __forceinline__ unsigned long long mg_zero(unsigned tag)
{
    return (unsigned long long)tag << 32;
}

__device__ __forceinline__ float mg_f(unsigned long long v)
{
    return __uint_as_float((unsigned)v);
}

// Whether a wait of this block has run out (set to 0 at the kernel's start).
__device__ __forceinline__ int &mg_gave_up()
{
    __shared__ int flag;
    return flag;
}

// The same answer in every lane of the warp.
__device__ __forceinline__ bool mg_give_up(long long polls, int *status)
{
    if ((polls & 15) != 0) return false;
    const bool quit = polls > kMgPollLimit || (*(volatile int *)status & MPMG_DEV_ERR_SPIN) != 0;
    if (!__any_sync(0xffffffffu, quit)) return false;
    atomicOr(status, MPMG_DEV_ERR_SPIN);
    mg_gave_up() = 1;
    return true;
}

// Waits until every word of v carries `tag` (addr(t, q) is the address of
// word q of trip t, for T trips of Q words).  Called by whole warps.  While some
// lane holds stale words, every lane loads its stale words again, kMgNap ns
// after the last round: the staged phases wait for a thousand words a block at
// most, so this floods nothing, and a word is in a register one round trip
// after it is visible (one lane polling one word and the rest reloaded after
// it cost a second round trip: 0.456 against 0.441 ms a step on the 130^2
// silo).  Bounded (kMgPollLimit polls, or another block's timeout): then the
// spin error is set, the words read NaN and the answer is false.
template <int T, int Q, class Addr>
__device__ __forceinline__ bool mg_resolve(unsigned long long (&v)[T][Q], unsigned tag, int *status, Addr addr)
{
    for (long long polls = 1;; polls++) {
        bool stale = false;
#pragma unroll
        for (int t = 0; t < T; t++) {
#pragma unroll
            for (int q = 0; q < Q; q++) stale |= (unsigned)(v[t][q] >> 32) != tag;
        }
        if (!__any_sync(0xffffffffu, stale)) return true;
        if (mg_give_up(polls, status)) {
#pragma unroll
            for (int t = 0; t < T; t++) {
#pragma unroll
                for (int q = 0; q < Q; q++) v[t][q] = mg_zero(tag) | 0x7fffffffu;
            }
            return false;
        }
        __nanosleep(kMgNap);
#pragma unroll
        for (int t = 0; t < T; t++) {
#pragma unroll
            for (int q = 0; q < Q; q++) {
                if ((unsigned)(v[t][q] >> 32) != tag) v[t][q] = mg_ld(addr(t, q));
            }
        }
    }
}

// Copies the words of two node ranges of a level vector (nn nodes), [a0, a1)
// to d0 and [b0, b1) to d1, as floats once they carry `tag`; nodes outside
// the level read 0.  Called by the whole block; ends with a block barrier.
__device__ __noinline__ void mg_stage(const unsigned long long *w, int nn, int a0, int a1, float *d0, int b0,
                                         int b1, float *d1, unsigned tag, int *status)
{
    constexpr int T = 4;
    const int na = max(a1 - a0, 0), nt = na + max(b1 - b0, 0);
    for (int base = 0; base < nt; base += T * kMgThreads) {
        unsigned long long v[T][1];
#pragma unroll
        for (int t = 0; t < T; t++) {
            const int u = base + threadIdx.x + t * kMgThreads;
            const int m = u < na ? a0 + u : b0 + (u - na);
            v[t][0] = (u < nt && m >= 0 && m < nn) ? mg_ld(w + m) : mg_zero(tag);
        }
        mg_resolve(v, tag, status, [&](int t, int) {
            const int u = base + threadIdx.x + t * kMgThreads;
            return w + (u < na ? a0 + u : b0 + (u - na));
        });
#pragma unroll
        for (int t = 0; t < T; t++) {
            const int u = base + threadIdx.x + t * kMgThreads;
            if (u < na) d0[u] = mg_f(v[t][0]);
            else if (u < nt) d1[u - na] = mg_f(v[t][0]);
        }
    }
    __syncthreads();
}

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

// All-gather of the four per-block inner products of V-cycle `tag`: each block
// publishes its values as tagged words (a double as two), and warp c waits for
// value c of every block and adds them in block order (lane l the blocks l,
// l + 32, ..., then a shuffle tree).  A block goes on only when every block has
// published, and every block publishes after its last read of the V-cycle's
// words: this is the grid barrier between V-cycles too, in one round trip
// instead of an arrival, a release and a read.  Two buffers, by the V-cycle's
// parity: a block that runs ahead writes the next but one only after every
// block has published, hence read, the one between.
// A block with a wait that ran out in the V-cycle publishes NaN for the last
// value, the residual, so that no block converges on that cycle.  False, in
// every thread, where the wait here runs out: v is not to be used then.
__device__ __forceinline__ bool mg_gather4(const mat::Unit &u, unsigned long long *words, double v[4], int nblocks,
                                           double *scratch, unsigned tag, int *status)
{
    const int nt = blockDim.x;
    bool ok = true;
    if (threadIdx.x < 4) {
        unsigned long long b = (unsigned long long)__double_as_longlong(
            threadIdx.x == 0 ? v[0] : threadIdx.x == 1 ? v[1] : threadIdx.x == 2 ? v[2] : v[3]);
        if (threadIdx.x == 3 && mg_gave_up() != 0) b = ~0ull;      // NaN
        unsigned long long *w = words + 2 * ((size_t)threadIdx.x * nblocks + blockIdx.x);
        const unsigned long long t = (unsigned long long)tag << 32;
        asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(w), "l"(t | (b & 0xffffffffu)));
        asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(w + 1), "l"(t | (b >> 32)));
    }
    if (threadIdx.x < 128) {
        const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
        constexpr int kMax = kMgBlocks / 32;
        unsigned long long p[kMax][2];
        const unsigned long long *base = words + 2 * (size_t)c * nblocks;
#pragma unroll
        for (int q = 0; q < kMax; q++) {
            const int t = lane + 32 * q;
#pragma unroll
            for (int h = 0; h < 2; h++) p[q][h] = t < nblocks ? mg_ld(base + 2 * t + h) : mg_zero(tag);
        }
        ok = mg_resolve(p, tag, status, [&](int q, int h) { return base + 2 * (lane + 32 * q) + h; });
        double x = 0;
#pragma unroll
        for (int q = 0; q < kMax; q++)
            if (32 * q < nblocks)
                x = u.add(x, __longlong_as_double((long long)((p[q][1] << 32) | (p[q][0] & 0xffffffffu))));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) x = u.add(x, __shfl_down_sync(0xffffffffu, x, off));
        if (lane == 0) scratch[4 * nt + c] = x;
    }
    const bool failed = __syncthreads_or(!ok);
#pragma unroll
    for (int c = 0; c < 4; c++) v[c] = scratch[4 * nt + c];
    __syncthreads();
    return !failed;
}
