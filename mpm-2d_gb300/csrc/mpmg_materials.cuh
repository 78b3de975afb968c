// Per-particle constitutive updates as device functions.  Each follows its
// reference plugin line by line; products, sums and quotients use the _rn
// intrinsics so that nvcc cannot fuse them into multiply-adds, which keeps
// the results bit-identical to the reference compiled without contraction.
#pragma once

#include "mpmg_internal.cuh"

namespace mat {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dadd_rn(a, -b); }

// a / b where the divisor b is fixed for the run and y = RN(1 / b) was
// formed once on the host.  Markstein's correction q' = RN(q + r y), with the
// residual r = a - b q exact through an FMA, is applied twice from q = RN(a y):
// the first brings q within one ulp of a / b, and from there the second
// returns the correctly rounded quotient (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34(1), 1990).  Five FP64 operations in place of a full division; the
// result equals a / b for normal operands and quotients (a zero quotient
// comes out +0, and non-finite operands are not carried through).  The laws
// divide by dvd_const below, in no FP64 operation; this form is kept as the
// five-operation alternative that tests/test_gpu_arith.py measures.
__device__ __forceinline__ double dvd_known(double a, double b, double y)
{
    double q = __dmul_rn(a, y);
    double r = __fma_rn(-b, q, a);
    q = __fma_rn(r, y, q);
    r = __fma_rn(-b, q, a);
    return __fma_rn(r, y, q);
}

// A divisor b fixed for the run: 1 / |b| = Z 2^(ez - 64) with Z the top 64
// bits (truncated) of the reciprocal, formed on the host.
struct Known {
    double b;
    uint64_t Z;
    int ez;                 // exponent of 1 / |b| (out of every range where b is not moderate)
};

inline Known make_known(double b)
{
    Known k;
    k.b = b;
    k.Z = 0;
    k.ez = 1 << 20;
    const double m = fabs(b);
    if (!(m > 0x1p-400 && m < 0x1p400)) return k;
    int e;
    const uint64_t B = (uint64_t)ldexp(frexp(m, &e), 53);      // m = B 2^(e - 53), 2^52 <= B < 2^53
    // 2^116 / B in [2^63, 2^64]
    const unsigned __int128 z = ((unsigned __int128)1 << 116) / B;
    k.Z = (z >> 64) != 0 ? ~0ull : (uint64_t)z;                // B = 2^52: 2^64 - 1 stands for 2^64
    k.ez = 1 - e;
    return k;
}

// The compiler's operations, out of line: the rare operands the shortcuts
// below leave to them.  (Under a predicate instead of a branch they would cost
// the FP64 pipe what they cost when they run.)
static __device__ __noinline__ double div_ieee(double a, double b)
{
    return __ddiv_rn(a, b);
}
static __device__ __noinline__ double mul_ieee(double a, double b)
{
    return __dmul_rn(a, b);
}
static __device__ __noinline__ double sqrt_ieee(double a)
{
    return __dsqrt_rn(a);
}

// a / b correctly rounded without an FP64 operation.  With a's 53-bit
// significand at the top of A and Z truncated, the exact quotient's 64-bit
// significand lies in [P, P + 2), P the high word of A Z, and in [P, P + 4)
// after the normalising shift.  Its 11 bits below the double's decide the
// rounding (a quotient is never a midpoint) unless they are within 4 of half:
// those four patterns of 2048, and operands or results outside the normal
// range, take the compiler's division.  A zero is returned as one.
__device__ __forceinline__ double dvd_const(double a, const Known &k)
{
    const int hi = __double2hiint(a), lo = __double2loint(a);
    const int e = (hi >> 20) & 0x7ff;
    const uint64_t A = ((uint64_t)(uint32_t)((hi & 0xfffff) | 0x100000) << 32 | (uint32_t)lo) << 11;
    uint64_t P = __umul64hi(A, k.Z);
    const int s = (int)(P >> 63) ^ 1;
    P <<= s;
    const int low = (int)P & 0x7ff, er = e + k.ez - s;
    const int sign = (hi ^ __double2hiint(k.b)) & (int)0x80000000;
    if ((unsigned)(e - 1) >= 2046u || (unsigned)(er - 1) >= 2046u || (unsigned)(low - 0x3fc) < 4u) {
        if (((hi << 1) | lo) == 0 && k.Z != 0) return __hiloint2double(sign, 0);
        return div_ieee(a, k.b);
    }
    const uint64_t m = (P >> 11) + (uint64_t)(low >> 10) + ((uint64_t)(uint32_t)(er - 1) << 52);
    return __hiloint2double((int)(m >> 32) | sign, (int)m);
}

// RN(a b) in integer arithmetic: the FP64 pipe issues one instruction a warp in
// 64 cycles and bounds the kernels that use this, while their integer pipe
// idles, and a product takes about 40 integer instructions.  With both
// significands at the top of 64 bits the exact product's upper 64 bits lie in
// [P, P + 3), P the high parts of three of the four 32-bit products, and in
// [P, P + 6) after the normalising shift; the 11 bits below the double's
// decide the rounding unless they lie next to half (six patterns of 2048, a
// tie among them).  Those, and operands outside 2^-255 .. 2^256 (zeros, for
// one), take the FP64 instruction.
__device__ __forceinline__ double imul(double a, double b)
{
    const int ha = __double2hiint(a), hb = __double2hiint(b);
    const unsigned la = (unsigned)__double2loint(a), lb = (unsigned)__double2loint(b);
    const unsigned Ah = __funnelshift_l(la, (unsigned)ha, 11) | 0x80000000u, Al = la << 11;
    const unsigned Bh = __funnelshift_l(lb, (unsigned)hb, 11) | 0x80000000u, Bl = lb << 11;
    const unsigned ea = (unsigned)(ha & 0x7ff00000) - (768u << 20), eb = (unsigned)(hb & 0x7ff00000) - (768u << 20);
    unsigned long long P = (unsigned long long)Ah * Bh + __umulhi(Ah, Bl) + __umulhi(Al, Bh);
    const unsigned up = (unsigned)(P >> 63);
    P <<= up ^ 1u;
    const unsigned low = (unsigned)P & 0x7ffu;
    if ((ea | eb) >= (512u << 20) || low - 0x3fbu < 6u) return mul_ieee(a, b);
    const unsigned long long m = (P >> 11) + (low >> 10);
    // biased exponents 768 + x and 768 + y give 513 + x + y (the significand's
    // leading one adds the rest)
    const unsigned e = ea + eb + (512u << 20) + (up << 20);
    return __hiloint2double((int)((unsigned)(m >> 32) + e + ((unsigned)(ha ^ hb) & 0x80000000u)), (int)(unsigned)m);
}

// Sign and order tests on the bit patterns (the FP64 pipe issues a compare at
// the rate of a multiply): non-negative doubles order as integers.
__device__ __forceinline__ bool is_nan(double a)
{
    return (__double_as_longlong(a) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool is_pos(double a)   // a > 0
{
    const long long b = __double_as_longlong(a);
    return b > 0 && b <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool is_neg(double a)   // a < 0
{
    const long long b = __double_as_longlong(a);
    return b > (long long)0x8000000000000000ULL && b <= (long long)0xfff0000000000000ULL;
}
__device__ __forceinline__ bool less_equal_pos(double a, double b)   // a <= b for a >= +0 or NaN, b not -0
{
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    return x >= 0 && x <= y && y <= 0x7ff0000000000000LL;
}
__device__ __forceinline__ bool is_finite(double a)
{
    return (__double2hiint(a) & 0x7ff00000) != 0x7ff00000;
}

// IEEE square root and quotient in one FP64 operation.  GB300's FP64 pipe runs
// at 1/64 of its FP32 rate and bounds the kernels that use these, while the
// integer and FP32 pipes idle: so all but the residual is formed there.  The
// operand's 52-bit significand is split into an FP32 head and tail, the
// approximate FP32 reciprocal (root) gives the result's head, and the head's
// residual, exact in an FP32 FMA, its tail: head + tail is good to about 2^-44
// and is assembled into a double by integer addition (the head held in [1, 2],
// where the double's spacing is one).  The exact residual of that double (the
// one FP64 FMA) times the FP32 reciprocal is the rest of the result in units
// of its last place, at most 512 of them and known to 2^-12: its nearest
// integer is added to the bit pattern.  The result is then the correctly
// rounded one (a square root or quotient of doubles is never a midpoint)
// unless the rest lies within 2^-11 of half a unit (one operand in 1024): those,
// results at the ends of a binade, zeros, negatives, non-finite values and
// exponents near the ends of the range take the compiler's operation.  That
// one issues eight FP64 instructions; with these, the integer quotients by
// constants and products above and the integer compares, the G2P with
// g_local_mu2 issues 72 FP64 instructions a warp of particles (211 with the
// compiler's operations): 156 us at 1 048 576 particles, 417 with those.

// The FP32 head (in [1, 2)) and tail of a double's significand.
__device__ __forceinline__ float sig_head(int hi, int lo, int exponent)
{
    return __int_as_float(((127 + exponent) << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)lo >> 29));
}
__device__ __forceinline__ float sig_tail(int lo, float unit)   // to 23 bits, without a conversion
{
    return (__int_as_float(0x3f800000 | (lo & 0x1fffffff) >> 6) - 1.0f) * unit;
}
// The bits of the double with a normal float's value times 2^e.
__device__ __forceinline__ long long widen(float f, int e)
{
    const unsigned b = __float_as_uint(f);
    return __double_as_longlong(__hiloint2double((int)((b >> 3) + ((unsigned)(896 + e) << 20)), (int)(b << 29)));
}

// A non-negative integer as a double, in integer arithmetic (conversions run
// on the FP64 pipe).
__device__ __forceinline__ double small_int(int c)
{
    const int z = __clz(c);
    const unsigned m = (unsigned)c << (z & 31);
    return __hiloint2double(c == 0 ? 0 : (int)(((1022u + 31 - z) << 20) + (m >> 11)), c == 0 ? 0 : (int)(m << 21));
}

// A residual r times 2^e as FP32 (truncated; zero stays zero), for results of
// moderate exponent.
__device__ __forceinline__ float residual(double r, int e)
{
    const int hi = __double2hiint(r), lo = __double2loint(r);
    const int f = ((hi >> 20) & 0x7ff) + e;
    const int b = (hi & (int)0x80000000) | ((f - 896) << 23) | ((hi & 0xfffff) << 3) | (int)((unsigned)lo >> 29);
    return (unsigned)(f - 897) < 254u ? __int_as_float(b) : 0.0f;
}

// The bit pattern s0 moved by d units, or false where that does not decide the
// rounding or leaves the binade of exponent field f.
__device__ __forceinline__ bool settle(long long &s0, float d, int f)
{
    const float t = rintf(d);
    const long long s = s0 + (long long)(int)t;
    const bool ok = fabsf(d - t) <= 0.5f - 0x1p-11f && fabsf(d) < 512.0f && (int)(s0 >> 52) == f && (int)(s >> 52) == f;
    s0 = s;
    return ok;
}

// sqrt(2^E x).
template <int E = 0>
__device__ __forceinline__ double root(double x)
{
    static_assert(E == 0 || E == -1, "the fallback's factor");
    const int hi = __double2hiint(x) + (E << 20), lo = __double2loint(x);
    const double xs = __hiloint2double(hi, lo);
    const int e = (hi >> 20) - 1023, odd = e & 1, k = e >> 1;
    // x = m 4^k, m = head + tail in [1, 4)
    const float mh = sig_head(hi, lo, odd), ml = sig_tail(lo, odd ? 0x1p-22f : 0x1p-23f);
    const float y = rsqrtf(mh);
    const float sh = fminf(fmaxf(mh * y, 1.0f), 2.0f);
    const float sl = 0.5f * y * (__fmaf_rn(-sh, sh, mh) + ml);
    long long s = widen(sh, k) + ((long long)__float2int_rn(sl * 0x1p50f) << 2);
    const double s0 = __longlong_as_double(s);
    const double r = __fma_rn(-s0, s0, xs);
    // sqrt(x) - s0 = r / (2 s0), in units 2^(k - 52)
    const bool fine = settle(s, residual(r, 51 - 2 * k) * y, 1023 + k);
    if (!fine || (unsigned)__double2hiint(x) - (223u << 20) >= (1600u << 20))   // outside 2^-800 .. 2^800
        return sqrt_ieee(E == 0 ? x : __dmul_rn(x, 0.5));
    return __longlong_as_double(s);
}

// 2^E a / b.
template <int E = 0>
__device__ __forceinline__ double quot(double a, double b)
{
    static_assert(E == 0 || E == 1, "the fallback's factor");
    const int ah = (__double2hiint(a) & 0x7fffffff) + (E << 20), al = __double2loint(a);
    const int bh = __double2hiint(b) & 0x7fffffff, bl = __double2loint(b);
    const double am = __hiloint2double(ah, al), bm = __hiloint2double(bh, bl);
    const long long frac = 0xfffffffffffffLL;
    // significands scaled so that the quotient's lies in [1, 2)
    const int up = (__double_as_longlong(am) & frac) < (__double_as_longlong(bm) & frac) ? 1 : 0;
    const float afh = sig_head(ah, al, up), afl = sig_tail(al, up ? 0x1p-22f : 0x1p-23f);
    const float bfh = sig_head(bh, bl, 0), bfl = sig_tail(bl, 0x1p-23f);
    const float y = __fdividef(1.0f, bfh);
    const float qh = fminf(fmaxf(afh * y, 1.0f), 2.0f);
    const float ql = __fmaf_rn(-qh, bfl, __fmaf_rn(-qh, bfh, afh) + afl) * y;
    const int eb = (bh >> 20) - 1023, eq = (ah >> 20) - 1023 - eb - up;
    long long q = widen(qh, eq) + ((long long)__float2int_rn(ql * 0x1p50f) << 2);
    const double r = __fma_rn(-bm, __longlong_as_double(q), am);
    // a / b - q0 = r / b, in units 2^(eq - 52)
    const bool fine = settle(q, residual(r, 52 - eb - eq) * y, 1023 + eq);
    if (!fine || (unsigned)((ah >> 20) - 624) >= 799u || (unsigned)((bh >> 20) - 624) >= 799u)   // 2^-399 .. 2^399
        return div_ieee(E == 0 ? a : __dmul_rn(a, 2.0), b);
    const int sign = (__double2hiint(a) ^ __double2hiint(b)) & (int)0x80000000;
    return __hiloint2double((int)(q >> 32) | sign, (int)q);
}

// Products, sums and constants for the FP64 pipe.  On GB300 a DFMA whose three
// operands are registers occupies a sub-partition's FP64 unit for 64.5 cycles;
// DADD, DMUL and any operand from the constant bank or an immediate cost 76.6,
// a compare 95.5 (measured, one to eight warps).  So the hot kernels form
// a b as a b + (-0) and a + b as a 1 + b (the same results bit for bit), and
// keep 1, -0 and every other constant in shared memory, from where they load
// into registers; as literals or kernel parameters the compiler would fold
// them back.  (It also folds a shared variable that only ever holds one
// constant: those are stored through opaque().)
__device__ __forceinline__ double opaque(double x)
{
    asm volatile("" : "+d"(x));
    return x;
}

struct Unit {
    double one, nz;         // 1, -0
    __device__ __forceinline__ double mul(double a, double b) const { return __fma_rn(a, b, nz); }
    __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(a, one, b); }
    __device__ __forceinline__ double sub(double a, double b) const { return __fma_rn(a, one, -b); }
};

struct Elastic : Unit {
    double G, K, lambda, dt;
    double twoG;            // 2 G, exact
    double Gdt;             // RN(G dt)
    double half, two, mfour;
    Known k3, kG, kdt, kGdt;     // 3, G, dt and RN(G dt) as divisors
};

// The same with integer products.
struct SoftElastic : Elastic {
    __device__ __forceinline__ double mul(double a, double b) const { return imul(a, b); }
};

inline Elastic make_elastic(double G, double K, double lambda, double dt)
{
    Elastic el;
    el.one = 1.0;
    el.nz = -0.0;
    el.G = G;
    el.K = K;
    el.lambda = lambda;
    el.dt = dt;
    el.twoG = 2.0 * G;
    el.Gdt = G * dt;
    el.half = 0.5;
    el.two = 2.0;
    el.mfour = -4.0;
    el.k3 = make_known(3.0);
    el.kG = make_known(G);
    el.kdt = make_known(dt);
    el.kGdt = make_known(el.Gdt);
    return el;
}

// exp(x) for the volume update v <- v exp(dt tr D), whose argument is tiny at
// any stable time step.  Where |x| < 2^-14 it is the degree-4 Taylor polynomial
// (truncation below x^5 / 120 < 2^-76) as a 64-bit integer in units of 2^-62,
// without an FP64 operation: x is shifted into place, x^2 / 2 is an integer
// product, and the rest, below 2^-44, comes from FP32 to 2^-66.  Where
// |x| < 2^-9 it is the degree-5 polynomial in Horner form (truncation below
// x^6 / 720 < 2^-63).  Either is within a hundredth of an ulp before its last
// rounding, so the result lies within about half an ulp of e^x; elsewhere exp().
static __device__ __noinline__ double exp_wide(double x)
{
    if ((__double2hiint(x) & 0x7fffffff) >= 0x3f600000) return exp(x);
    double p = __fma_rn(x, 1.0 / 120.0, 1.0 / 24.0);
    p = __fma_rn(p, x, 1.0 / 6.0);
    p = __fma_rn(p, x, 0.5);
    p = __fma_rn(p, x, 1.0);
    return __fma_rn(p, x, 1.0);
}

__device__ __forceinline__ double exp_small(double x)
{
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const int e = (hi >> 20) & 0x7ff;
    if (e >= 1023 - 14) return exp_wide(x);
    const unsigned long long sig =
        ((unsigned long long)(unsigned)((hi & 0xfffff) | 0x100000) << 32 | (unsigned)lo) << 11;
    // below 2^-62 x does not count
    const long long X = (long long)(sig >> min(1024 - e, 63));
    const float xf = __int_as_float((hi & (int)0x80000000) | (max(e, 960) - 896) << 23 | (hi & 0xfffff) << 3);
    const int w = __float2int_rn(xf * xf * xf * __fmaf_rn(xf, 1.0f / 24.0f, 1.0f / 6.0f) * 0x1p62f);
    const long long r = (1LL << 62) + (long long)__umul64hi(2 * X, X) + w + (hi < 0 ? -X : X);
    // rounded to 2^-52 from one upwards, to 2^-53 below
    const bool up = r >= 1LL << 62;
    const long long m = up ? (r + 512) >> 10 : (r + 256) >> 9;
    return __hiloint2double((int)(m >> 32) + ((up ? 1022 : 1021) << 20), (int)m);
}

// isolin calculate_stress_threaded, materialsrc/isolin.c:75-116.
template <class E>
__device__ __forceinline__ void isolin(const E &el, double exx, double exy, double eyy,
                                       double wxy, double &sxx, double &sxy, double &syy)
{
    const auto mul = [&](double a, double b) { return el.mul(a, b); };
    const auto add = [&](double a, double b) { return el.add(a, b); };
    const auto sub = [&](double a, double b) { return el.sub(a, b); };
    const double twoG = el.twoG;
    double trD = add(exx, eyy);
    double dsjxx = add(mul(el.lambda, trD), mul(twoG, exx));
    double dsjxy = mul(twoG, exy);
    double dsjyy = add(mul(el.lambda, trD), mul(twoG, eyy));
    const double ws = mul(wxy, sxy);   // 2 ws rides in the FMAs: the doubling is exact
    dsjxx = __fma_rn(el.two, ws, dsjxx);
    dsjxy = sub(dsjxy, mul(wxy, sub(sxx, syy)));
    dsjyy = __fma_rn(-el.two, ws, dsjyy);
    sxx = add(sxx, mul(el.dt, dsjxx));
    sxy = add(sxy, mul(el.dt, dsjxy));
    syy = add(syy, mul(el.dt, dsjyy));
}

// negative_root, g_local_mu2.c:90-99 (also g_nonlocal_mu2.c:226-235), with
// a = 1: the products by 4 and 2 are exact, so they ride in an FMA and in the
// quotient's exponent.
template <class E>
__device__ __forceinline__ double negative_root(const E &el, double b, double c)
{
    const double disc = root(__fma_rn(el.mfour, c, el.mul(b, b)));
    if (is_pos(b)) return el.mul(el.half, el.sub(-b, disc));
    return quot<1>(c, el.sub(disc, b));
}

struct Mu2Params {
    double mu_s, mu_2, I0, grains_rho, grains_d, rho_critical, A;
    Known krho, kd, kAAdd;                 // grains_rho, grains_d and A^2 d^2 as divisors
    double rho_lo, rho_hi;                 // RN(rho_critical (1 - 2^-47)), RN(rho_critical (1 + 2^-47)); -1 and
                                           // infinity (no bracket) where rho_critical is not in 2^-60 .. 2^60
    double alpha_c;                        // G I0 dt / (grains_d sqrt(grains_rho))
    double GI0dt;                          // RN(RN(G I0) dt), formed on the host
};

// RN(m / v) < rho_critical, decided as the reference's division and compare
// decide it, without the division for most particles.  For normal v > 0 and
// rho_lo, rho_hi as above: m < RN(v rho_lo) implies
// m / v < rho_critical (1 - 2^-48), hence RN(m / v) < rho_critical; and
// m > RN(v rho_hi) implies m / v > rho_critical (1 + 2^-48), hence
// RN(m / v) > rho_critical (the roundings add at most 3 2^-53 relative, and
// the doubles within 2^-48 of rho_critical are further than an ulp from it).
// Only m inside the bracket, and any operand that is not a normal positive
// number above 2^-959 (or a NaN), takes the division.  Positive normal
// products and m order as integers; the dense side is tested first.
template <class U>
__device__ __forceinline__ bool below_density(const U &u, double m, double v, const Mu2Params &mp)
{
    const long long mb = __double_as_longlong(m), vb = __double_as_longlong(v);
    if (vb > 0x0400000000000000LL && vb < 0x7ff0000000000000LL && mb > 0x0400000000000000LL &&
        mb < 0x7ff0000000000000LL) {
        if (mb > __double_as_longlong(u.mul(v, mp.rho_hi))) return false;
        if (mb < __double_as_longlong(u.mul(v, mp.rho_lo))) return true;
    }
    return __ddiv_rn(m, v) < mp.rho_critical;
}

// g_local_mu2 calculate_stress_threaded, g_local_mu2.c:165-310, written for
// the plane-strain stress it keeps: T = [[Txx, Txy, 0], [Txy, Tyy, 0],
// [0, 0, Tzz]] (the z-shear components stay zero and T stays symmetric
// because L has no z entries).  The expressions are the tensor.c sums with
// their zero terms removed, in the same order.
template <class E>
__device__ __forceinline__ void g_local_mu2(const E &el, const Mu2Params &mp, double m,
                                            double v, double exx, double eyy, double d2,
                                            double w2, double &Txx, double &Txy, double &Tyy,
                                            double &Tzz, double &gammap, double &gammadotp)
{
    const auto mul = [&](double a, double b) { return el.mul(a, b); };
    const auto add = [&](double a, double b) { return el.add(a, b); };
    const auto sub = [&](double a, double b) { return el.sub(a, b); };
    const double G = el.G, dt = el.dt;
    const double lambda = el.lambda;   // K - 2 G / 3, formed on the host with the same roundings
    // d2 = Lxy + Lyx = 2 Dxy, w2 = Lxy - Lyx = 2 Wxy (L :191-199, W = skw(L),
    // D = sym(L) tensor.c:330-384).
    // Exact shortcuts, bit for bit the reference's values for normal
    // operands below DBL_MAX / 2 (a halving or doubling commutes with a
    // rounding): 0.5 (x + x) is x; W T - T W has
    // xx entry RN(Wxy Txy) + RN(Wxy Txy) = RN(w2 Txy), yy entry its negative,
    // and xy entry half of RN(w2 Tyy) - RN(Txx w2), added with one rounding by
    // an FMA; Dxy 2G is d2 G; 0 * 2G is +0.
    const double trD = add(exx, eyy);
    // Jaumann term JS = W T - T W (:209-212)
    const double JSxx = mul(w2, Txy);
    const double JSxy2 = sub(mul(w2, Tyy), mul(Txx, w2));
    // trial stress (:215-222)
    const double twoG = el.twoG;
    const double lt = mul(lambda, trD);
    const double Txx_tr = add(mul(add(add(mul(exx, twoG), lt), JSxx), dt), Txx);
    const double Txy_tr = add(mul(__fma_rn(el.half, JSxy2, mul(d2, G)), dt), Txy);
    const double Tyy_tr = add(mul(sub(add(mul(eyy, twoG), lt), JSxx), dt), Tyy);
    const double Tzz_tr = add(mul(lt, dt), Tzz);
    // decompose and contract (:225-228; tensor.c:205-224, :422-437)
    double p_tr = dvd_const(add(add(Txx_tr, Tyy_tr), Tzz_tr), el.k3);
    const double T0xx = sub(Txx_tr, p_tr), T0xy = Txy_tr, T0yy = sub(Tyy_tr, p_tr), T0zz = sub(Tzz_tr, p_tr);
    const double xy2 = mul(T0xy, T0xy);
    const double tt = add(add(add(add(mul(T0xx, T0xx), xy2), xy2), mul(T0yy, T0yy)), mul(T0zz, T0zz));
    const double tau_tr = root<-1>(tt);
    p_tr = -p_tr;

    const bool density_flag = below_density(el, m, v, mp);
    double nup_tau;
    if (density_flag || !(is_pos(p_tr) || is_nan(p_tr))) {
        nup_tau = 0;
        Txx = 0; Txy = 0; Tyy = 0; Tzz = 0;
    } else if (is_pos(p_tr)) {
        const double S0 = mul(mp.mu_s, p_tr);
        if (less_equal_pos(tau_tr, S0)) {
            // tau_tau = tau_tr, scale factor 1: (tau_tr - tau_tau) / G / dt
            // is +0 and T0 * 1 is T0 exactly, so neither is formed
            nup_tau = is_finite(tau_tr) ? 0.0 : mul(sub(tau_tr, tau_tr), dt);
            Txx = sub(T0xx, p_tr);
            Txy = T0xy;
            Tyy = sub(T0yy, p_tr);
            Tzz = sub(T0zz, p_tr);
        } else {
            const double S2 = mul(mp.mu_2, p_tr);
            const double alpha = dvd_const(mul(mp.GI0dt, root(dvd_const(p_tr, mp.krho))), mp.kd);
            const double B = -add(add(S2, tau_tr), alpha);
            const double H = add(mul(S2, tau_tr), mul(S0, alpha));
            const double tau_tau = negative_root(el, B, H);
            const double scale_factor = quot(tau_tau, tau_tr);
            nup_tau = dvd_const(dvd_const(sub(tau_tr, tau_tau), el.kG), el.kdt);
            Txx = sub(mul(T0xx, scale_factor), p_tr);
            Txy = mul(T0xy, scale_factor);
            Tyy = sub(mul(T0yy, scale_factor), p_tr);
            Tzz = sub(mul(T0zz, scale_factor), p_tr);
        }
    } else {
        nup_tau = 0;   // NaN pressure: the reference prints 'u' and keeps T
    }
    gammap = add(gammap, mul(nup_tau, dt));
    gammadotp = nup_tau;
}

// The plane-stress-form local returns that share one structure:
//   dp_ri_mt                  dp_ri_mt.c:99-200                  3D trial, Drucker-Prager return
//   g_local_mu2_plane_strain  g_local_mu2_plane_strain.c:157-265 3D trial, mu(I) return, beta
//   g_local_mu2_true_2d       g_local_mu2_true_2d.c:157-260      2D trial, mu(I) return, beta
// A 3D trial carries the out-of-plane stress szz (state[1]) and takes
// p = -(sxx + syy + szz) / 3; the 2D trial takes p = -(sxx + syy) / 2.  The
// Drucker-Prager return caps tau at mu_s p; the mu(I) return takes the
// negative root of g_local_mu2's quadratic.  Dilute particles (m / v below
// the literal 1485.0f) and particles in tension drop their stress and record
// the whole trial shear as plastic flow, and the beta variants record
// -p / (K dt) in state[5].  state[9] accumulates the plastic strain and
// state[10] holds its rate.
struct ReturnParams {
    double mu_s, mu_2, I0, grains_rho, grains_d, rho_critical;
};

template <bool TRIAL3D, bool MU_I, bool BETA, class E>
__device__ __forceinline__ void plane_return(const E &el, const ReturnParams &rp, double m, double v,
                                             double exx, double exy, double eyy, double wxy, double &sxx,
                                             double &sxy, double &syy, double &szz, double &beta,
                                             double &gammap, double &gammadotp)
{
    const auto mul = [&](double a, double b) { return el.mul(a, b); };
    const auto add = [&](double a, double b) { return el.add(a, b); };
    const auto sub = [&](double a, double b) { return el.sub(a, b); };
    const double G = el.G, K = el.K, dt = el.dt;
    const double lambda = el.lambda;   // K - 2 G / 3, formed on the host with the same roundings
    const double twoG = el.twoG;
    double trD = add(exx, eyy);
    double dsjxx = add(mul(lambda, trD), mul(twoG, exx));
    double dsjxy = mul(twoG, exy);
    double dsjyy = add(mul(lambda, trD), mul(twoG, eyy));
    const double ws = mul(wxy, sxy);   // 2 ws rides in the FMAs: the doubling is exact
    dsjxx = __fma_rn(el.two, ws, dsjxx);
    dsjxy = sub(dsjxy, mul(wxy, sub(sxx, syy)));
    dsjyy = __fma_rn(-el.two, ws, dsjyy);
    double sxx_tr = add(sxx, mul(dt, dsjxx));
    double sxy_tr = add(sxy, mul(dt, dsjxy));
    double syy_tr = add(syy, mul(dt, dsjyy));
    double p_tr, t0zz = 0, szz_tr = 0;
    if (TRIAL3D) {
        szz_tr = add(szz, mul(mul(dt, lambda), trD));
        p_tr = dvd_const(-add(add(sxx_tr, syy_tr), szz_tr), el.k3);
    } else {
        p_tr = -mul(el.half, add(sxx_tr, syy_tr));
    }
    double t0xx = add(sxx_tr, p_tr), t0xy = sxy_tr, t0yy = add(syy_tr, p_tr);
    double tt = add(__fma_rn(el.two, mul(t0xy, t0xy), mul(t0xx, t0xx)), mul(t0yy, t0yy));
    if (TRIAL3D) {
        t0zz = add(szz_tr, p_tr);
        tt = add(tt, mul(t0zz, t0zz));
    }
    double tau_tr = root<-1>(tt);

    const bool density_flag = quot(m, v) < rp.rho_critical;
    double nup_tau;
    if (density_flag || p_tr <= 0) {
        nup_tau = dvd_const(tau_tr, el.kGdt);
        if (BETA) beta = quot(-p_tr, mul(K, dt));
        sxx = 0; sxy = 0; syy = 0;
        if (TRIAL3D) szz = 0;
    } else if (p_tr > 0) {
        double S0 = mul(rp.mu_s, p_tr);
        double tau_tau, scale_factor;
        if (tau_tr <= S0) {
            tau_tau = tau_tr;
            scale_factor = 1.0;
        } else if (MU_I) {
            double S2 = mul(rp.mu_2, p_tr);
            double alpha = quot(mul(mul(mul(G, rp.I0), dt), root(quot(p_tr, rp.grains_rho))), rp.grains_d);
            double B = -add(add(S2, tau_tr), alpha);
            double H = add(mul(S2, tau_tr), mul(S0, alpha));
            tau_tau = negative_root(el, B, H);
            scale_factor = quot(tau_tau, tau_tr);
        } else {
            tau_tau = S0;
            scale_factor = quot(tau_tau, tau_tr);
        }
        nup_tau = dvd_const(dvd_const(sub(tau_tr, tau_tau), el.kG), el.kdt);
        if (BETA) beta = 0;
        sxx = sub(mul(scale_factor, t0xx), p_tr);
        sxy = mul(scale_factor, t0xy);
        syy = sub(mul(scale_factor, t0yy), p_tr);
        if (TRIAL3D) szz = sub(mul(scale_factor, t0zz), p_tr);
    } else {
        nup_tau = 0;   // NaN pressure: the reference prints 'u' and keeps s
    }
    gammap = add(gammap, mul(nup_tau, dt));
    gammadotp = nup_tau;
}

// g_local_mu2_reverse calculate_stress_threaded, g_local_mu2_reverse.c:166-302:
// a rate-dependent return to mu(I) (p + c), c = 0, with mu from the previous
// step's gammadotp and the start-of-step pressure, and Jaumann terms of the
// opposite sign to isolin's.  beta in state[5].
template <class E>
__device__ __forceinline__ void g_local_mu2_reverse(const E &el, const Mu2Params &mp, double m, double v,
                                                    double exx, double exy, double eyy, double wxy, double &sxx,
                                                    double &sxy, double &syy, double &beta, double &gammap,
                                                    double &gammadotp)
{
    const auto mul = [&](double a, double b) { return el.mul(a, b); };
    const auto add = [&](double a, double b) { return el.add(a, b); };
    const auto sub = [&](double a, double b) { return el.sub(a, b); };
    const double K = el.K, dt = el.dt, c = 0;
    const double lambda = el.lambda;
    const double twoG = el.twoG;
    double p_t = -mul(el.half, add(sxx, syy));
    double trD = add(exx, eyy);
    double dsjxx = add(mul(lambda, trD), mul(twoG, exx));
    double dsjxy = mul(twoG, exy);
    double dsjyy = add(mul(lambda, trD), mul(twoG, eyy));
    const double ws = mul(wxy, sxy);   // 2 ws rides in the FMAs: the doubling is exact
    dsjxx = __fma_rn(-el.two, ws, dsjxx);
    dsjxy = add(dsjxy, mul(wxy, sub(sxx, syy)));
    dsjyy = __fma_rn(el.two, ws, dsjyy);
    double sxx_tr = add(sxx, mul(dt, dsjxx));
    double sxy_tr = add(sxy, mul(dt, dsjxy));
    double syy_tr = add(syy, mul(dt, dsjyy));
    double p_tr = -mul(el.half, add(sxx_tr, syy_tr));
    double t0xx = add(sxx_tr, p_tr), t0xy = sxy_tr, t0yy = add(syy_tr, p_tr);
    double tau_tr = root<-1>((add(__fma_rn(el.two, mul(t0xy, t0xy), mul(t0xx, t0xx)), mul(t0yy, t0yy))));
    double inum = mul(mul(gammadotp, mp.grains_d), root(mp.grains_rho));
    double mu_t;
    if (p_t <= 0) {
        mu_t = mp.mu_2;
    } else {
        inum = quot(inum, root(p_t));
        if (inum <= 0) mu_t = mp.mu_s;
        else mu_t = add(mp.mu_s, quot(sub(mp.mu_2, mp.mu_s), add(quot(mp.I0, inum), 1.0)));
    }
    double tau_tau = mul(mu_t, add(p_tr, c));
    double f = sub(tau_tr, tau_tau);
    const bool density_flag = quot(m, v) < mp.rho_critical;
    const double pmin = quot(-c, mu_t);
    double nup_tau;
    if (density_flag) {
        nup_tau = dvd_const(tau_tr, el.kGdt);
        beta = quot(-p_tr, mul(K, dt));
        sxx = 0; sxy = 0; syy = 0;
    } else if (f < 0) {
        nup_tau = 0;
        beta = 0;
        sxx = sub(t0xx, p_tr);
        sxy = t0xy;
        syy = sub(t0yy, p_tr);
    } else if (f >= 0 && p_tr > pmin) {
        nup_tau = dvd_const(dvd_const(f, el.kG), el.kdt);
        beta = 0;
        double scale_factor = quot(tau_tau, tau_tr);
        sxx = sub(mul(scale_factor, t0xx), p_tr);
        sxy = mul(scale_factor, t0xy);
        syy = sub(mul(scale_factor, t0yy), p_tr);
    } else if (p_tr <= pmin) {
        nup_tau = dvd_const(tau_tr, el.kGdt);
        beta = quot(sub(quot(c, mu_t), p_tr), mul(K, dt));
        sxx = 0; sxy = 0; syy = 0;
    } else {
        nup_tau = 0;   // NaN: the reference prints the particle and keeps s
    }
    gammap = add(gammap, mul(nup_tau, dt));
    gammadotp = nup_tau;
}

// mu_from_gammadot, g_local_mu2_ext.c:75-95.
__device__ __forceinline__ double mu_from_gammadot(double gammadot, double p, double dsqrtrhos, double mu_s,
                                                   double mu_2, double inum_0)
{
    if (p <= 0) return mu_2;
    double inum = quot(mul(dsqrtrhos, gammadot), root(p));
    if (inum <= 0) return mu_s;
    return add(mu_s, quot(sub(mu_2, mu_s), add(quot(inum_0, inum), 1.0)));
}

// g_local_mu2_ext, first phase (g_local_mu2_ext.c:214-230): the local
// fluidity gammadotp / mu_t from the start-of-step pressure.  mu_t keeps its
// previous value where gammadotp is 0.
__device__ __forceinline__ void ext_local_fluidity(const Mu2Params &mp, double sxx, double syy, double gammadotp,
                                                   double &mu_t, double &gflocal)
{
    double p_t = mul(-0.5, add(sxx, syy));
    if (gammadotp == 0) {
        gflocal = 0;
    } else {
        mu_t = mu_from_gammadot(gammadotp, p_t, mul(mp.grains_d, root(mp.grains_rho)), mp.mu_s, mp.mu_2,
                                mp.I0);
        gflocal = quot(gammadotp, mu_t);
    }
}

// g_local_mu2_ext, third phase (g_local_mu2_ext.c:292-368): plane-stress
// elastic trial with the Jaumann terms, returned to mu(gammadotp) (p + c)
// with c = 1e-2.
__device__ __forceinline__ void ext_stress(const Elastic &el, const Mu2Params &mp, double E, double nu, double m,
                                           double v, double exx, double exy, double eyy, double wxy, double &sxx,
                                           double &sxy, double &syy, double &mu_t, double &beta, double &gammap,
                                           double &gammadotp)
{
    const auto mul = [&](double a, double b) { return el.mul(a, b); };
    const auto add = [&](double a, double b) { return el.add(a, b); };
    const auto sub = [&](double a, double b) { return el.sub(a, b); };
    const double K = el.K, dt = el.dt, c = 1e-2;
    double p_t = -mul(el.half, add(sxx, syy));
    const double Ep = quot(E, sub(el.one, mul(nu, nu)));
    const double Gp = quot(E, mul(el.two, add(el.one, nu)));
    double dsjxx = mul(mul(dt, Ep), add(exx, mul(nu, eyy)));
    double dsjxy = mul(mul(dt, Gp), exy);
    double dsjyy = mul(mul(dt, Ep), add(eyy, mul(nu, exx)));
    double w2 = mul(mul(mul(el.two, dt), wxy), sxy);
    dsjxx = sub(dsjxx, w2);
    dsjxy = add(dsjxy, mul(mul(dt, wxy), sub(sxx, syy)));
    dsjyy = add(dsjyy, w2);
    double sxx_tr = add(sxx, dsjxx), sxy_tr = add(sxy, dsjxy), syy_tr = add(syy, dsjyy);
    double p_tr = -mul(el.half, add(sxx_tr, syy_tr));
    double t0xx = add(sxx_tr, p_tr), t0xy = sxy_tr, t0yy = add(syy_tr, p_tr);
    double tau_tr = root<-1>((add(__fma_rn(el.two, mul(t0xy, t0xy), mul(t0xx, t0xx)), mul(t0yy, t0yy))));
    mu_t = mu_from_gammadot(gammadotp, p_t, mul(mp.grains_d, root(mp.grains_rho)), mp.mu_s, mp.mu_2, mp.I0);
    double tau_tau = mul(mu_t, add(p_tr, c));
    double f = sub(tau_tr, tau_tau);
    const bool density_flag = quot(m, v) < mp.rho_critical;
    const double pmin = quot(-c, mu_t);   // -c / mu_t, the reference's -c/mu_t
    double nup_tau;
    if (density_flag) {
        nup_tau = dvd_const(tau_tr, el.kGdt);
        beta = quot(-p_tr, mul(K, dt));
        sxx = 0; sxy = 0; syy = 0;
    } else if (f < 0) {
        nup_tau = 0;
        beta = 0;
        sxx = sub(t0xx, p_tr);
        sxy = t0xy;
        syy = sub(t0yy, p_tr);
    } else if (f >= 0 && p_tr > pmin) {
        nup_tau = dvd_const(sub(tau_tr, tau_tau), el.kGdt);
        beta = 0;
        double scale_factor = quot(tau_tau, tau_tr);
        sxx = sub(mul(scale_factor, t0xx), p_tr);
        sxy = mul(scale_factor, t0xy);
        syy = sub(mul(scale_factor, t0yy), p_tr);
    } else if (p_tr <= pmin) {
        nup_tau = dvd_const(tau_tr, el.kGdt);
        beta = quot(sub(quot(c, mu_t), p_tr), mul(K, dt));
        sxx = 0; sxy = 0; syy = 0;
    } else {
        nup_tau = 0;   // NaN: the reference prints the particle and keeps s
    }
    gammap = add(gammap, mul(nup_tau, dt));
    gammadotp = nup_tau;
}

// Trial Jaumann stress of g_nonlocal_mu2.c:166-186 (and :271-290), with
// lambda = K - 2G/3 (the reference leaves it uninitialised at :154).
template <class E>
__device__ __forceinline__ void nonlocal_mu2_trial(const E &el, double exx, double exy,
                                                   double eyy, double wxy, double sxx, double sxy,
                                                   double syy, double &p_tr, double &t0xx,
                                                   double &t0xy, double &t0yy, double &tau_tr)
{
    const auto mul = [&](double a, double b) { return el.mul(a, b); };
    const auto add = [&](double a, double b) { return el.add(a, b); };
    const auto sub = [&](double a, double b) { return el.sub(a, b); };
    const double dt = el.dt;
    const double lambda = el.lambda;   // sub(K, quot(mul(2, G), 3)), formed on the host with the same roundings
    const double twoG = el.twoG;
    double trD = add(exx, eyy);
    double dsjxx = add(mul(lambda, trD), mul(twoG, exx));
    double dsjxy = mul(twoG, exy);
    double dsjyy = add(mul(lambda, trD), mul(twoG, eyy));
    const double ws = mul(wxy, sxy);   // 2 ws rides in the FMAs: the doubling is exact
    dsjxx = __fma_rn(el.two, ws, dsjxx);
    dsjxy = sub(dsjxy, mul(wxy, sub(sxx, syy)));
    dsjyy = __fma_rn(-el.two, ws, dsjyy);
    double sxx_tr = add(sxx, mul(dt, dsjxx));
    double sxy_tr = add(sxy, mul(dt, dsjxy));
    double syy_tr = add(syy, mul(dt, dsjyy));
    p_tr = -mul(el.half, add(sxx_tr, syy_tr));
    t0xx = add(sxx_tr, p_tr);
    t0xy = sxy_tr;
    t0yy = add(syy_tr, p_tr);
    tau_tr = root<-1>((add(__fma_rn(el.two, mul(t0xy, t0xy), mul(t0xx, t0xx)), mul(t0yy, t0yy))));
}

// calculate_bulk_granular_fluidity, g_nonlocal_mu2.c:238-321, for one
// particle, from its trial pressure and shear stress (nonlocal_mu2_trial):
// dense flag, local fluidity and the inverse squared cooperativity length.
// The dense flag and the branches are the reference's decisions on the same
// values.  The flowing branch is the same algebra in fewer FP64 operations
// (these values feed the iterative fluidity solve, not a bit-exact output):
//   alpha    = G I0 dt sqrt(p / rho) / d  = alpha_c sqrt(p)
//   tau_tau  = the negative root of t^2 - B t + H, B = S2 + tau + alpha > 0,
//              as 2 H / (B + sqrt(B^2 - 4 H)) (negative_root's b < 0 branch)
//   gf_local = (p / (G dt)) (tau / tau_tau - 1) = p (tau - tau_tau) / (G dt tau_tau)
// and below yield (scale factor 1) gf_local is +0.
template <class E>
__device__ __forceinline__ void nonlocal_mu2_bulk(const E &el, const Mu2Params &mp, double m,
                                                  double v, double p_tr, double tau_tr, double &dense,
                                                  double &gf_local, double &xisq_inv)
{
    const auto mul = [&](double a, double b) { return el.mul(a, b); };
    const auto add = [&](double a, double b) { return el.add(a, b); };
    const auto sub = [&](double a, double b) { return el.sub(a, b); };
    const bool is_dense = !(below_density(el, m, v, mp) || is_neg(p_tr));
    dense = is_dense ? 1.0 : 0.0;
    if (!is_dense || !(is_pos(p_tr) || is_nan(p_tr))) {
        gf_local = 0;
        xisq_inv = 0;
    } else if (is_pos(p_tr)) {
        double tau_tau;
        double S0 = mul(mp.mu_s, p_tr);
        if (less_equal_pos(tau_tr, S0)) {
            tau_tau = tau_tr;
            gf_local = 0;
        } else {
            double S2 = mul(mp.mu_2, p_tr);
            double alpha = mul(mp.alpha_c, root(p_tr));
            double B = add(add(S2, tau_tr), alpha);
            double H = add(mul(S2, tau_tr), mul(S0, alpha));
            tau_tau = quot<1>(H, add(B, root(__fma_rn(el.mfour, H, mul(B, B)))));
            gf_local = quot(mul(p_tr, sub(tau_tr, tau_tau)), mul(el.Gdt, tau_tau));
        }
        xisq_inv = dvd_const(fabs(sub(quot(tau_tau, p_tr), mp.mu_s)), mp.kAAdd);
    } else {
        gf_local = 0;
        xisq_inv = 0;
    }
}

// Stress update after the fluidity solve, g_nonlocal_mu2.c:160-218. The
// reference forms the trial stress again at :166-186 from the same strain
// rates and start-of-step stress as the bulk pass; the G2P keeps that trial
// instead, with the dense flag folded into the pressure (p_d = p_tr where the
// particle is dense, 0 where it is not), so `dense == 0 || p_tr <= 0` reads
// `p_d <= 0`. sxx, sxy, syy hold the start-of-step stress, which a NaN trial
// pressure keeps (neither branch of the reference is taken).
template <class E>
__device__ __forceinline__ void nonlocal_mu2_stress(const E &el, double gf, double p_d,
                                                    double t0xx, double t0xy, double t0yy,
                                                    double tau_tr, double &sxx, double &sxy,
                                                    double &syy, double &gammap, double &gammadotp)
{
    const double p_tr = p_d;
    double nup_tau;
    if (!is_pos(p_tr) && !is_nan(p_tr)) {
        nup_tau = 0;
        sxx = 0; sxy = 0; syy = 0;
    } else if (is_pos(p_tr)) {
        const double scale_factor = quot(p_tr, el.add(el.mul(el.Gdt, gf), p_tr));
        const double tau_tau = el.mul(tau_tr, scale_factor);
        // ((tau - tau_tau) / G) / dt as one quotient by G dt (the fluidity
        // comes from an iterative solve, so this value is not bit-exact
        // with the reference's anyway)
        nup_tau = dvd_const(el.sub(tau_tr, tau_tau), el.kGdt);
        sxx = el.sub(el.mul(scale_factor, t0xx), p_tr);
        sxy = el.mul(scale_factor, t0xy);
        syy = el.sub(el.mul(scale_factor, t0yy), p_tr);
    } else {
        nup_tau = 0;
    }
    gammap = el.add(gammap, el.mul(nup_tau, el.dt));
    gammadotp = nup_tau;
}

struct NonlocalParams {
    double E, nu, mu_s, grains_rho, B, A, grains_d, cohesion;
};

// calculate_bulk_granular_fluidity, g_nonlocal.c:306-352, for one particle
// (the reference applies it to every particle, active or not).
__device__ __forceinline__ void nonlocal_bulk(const NonlocalParams &np, double sxx, double sxy,
                                              double syy, double &eta, double &gf_bulk,
                                              double &xisq_inv)
{
    const double p_cap = 1e-2;
    double p_t = mul(-0.5, add(sxx, syy));
    double a = add(sxx, p_t), b = sxy, c = add(syy, p_t);
    double tau_t = root<-1>((add(add(mul(a, a), mul(mul(2.0, b), b)), mul(c, c))));
    if (p_t < p_cap) p_t = p_cap;
    double S0 = mul(p_t, np.mu_s);
    eta = mul(mul(np.B, np.grains_d), root(mul(p_t, np.grains_rho)));
    xisq_inv = quot(fabs(sub(quot(tau_t, p_t), np.mu_s)),
                   mul(mul(mul(np.grains_d, np.grains_d), np.A), np.A));
    gf_bulk = (tau_t > S0) ? mul(quot(p_t, eta), sub(1.0, quot(S0, tau_t))) : 0.0;
}

// Explicit stress update of g_nonlocal.c:154-298 (every particle).
__device__ __forceinline__ void nonlocal_stress(const NonlocalParams &np, double G, double dt,
                                                double t, double gf, double exx, double exy,
                                                double eyy, double wxy, double &sxx, double &sxy,
                                                double &syy, double &gammap)
{
    const double EMOD = np.E, NUMOD = np.nu, c = np.cohesion;
    const double cA = quot(EMOD, sub(1.0, mul(NUMOD, NUMOD)));
    const double cB = quot(EMOD, mul(2.0, add(1.0, NUMOD)));
    double p_t = mul(-0.5, add(sxx, syy));
    double a = add(sxx, p_t), b = sxy, cc = add(syy, p_t);
    double tau_t;
    double dsjxx = mul(mul(dt, cA), add(exx, mul(NUMOD, eyy)));
    double dsjxy = mul(mul(dt, cB), exy);
    double dsjyy = mul(mul(dt, cA), add(eyy, mul(NUMOD, exx)));
    double jw = mul(mul(mul(2.0, dt), wxy), sxy);
    dsjxx = sub(dsjxx, jw);
    dsjxy = add(dsjxy, mul(mul(dt, wxy), sub(sxx, syy)));
    dsjyy = add(dsjyy, jw);
    double p_tr = mul(-0.5, add(add(sxx, dsjxx), add(syy, dsjyy)));
    if (p_tr < c) {
        sxx = quot(mul(0.5, c), np.mu_s);
        sxy = 0;
        syy = quot(mul(0.5, c), np.mu_s);
        return;
    }
    tau_t = root<-1>((add(add(mul(a, a), mul(mul(2.0, b), b)), mul(cc, cc))));
    const double r = root(0.5);
    double Npxx = quot(mul(r, a), tau_t);
    double Npxy = quot(mul(r, b), tau_t);
    double Npyy = quot(mul(r, cc), tau_t);
    double dxx0 = mul(0.5, sub(exx, eyy)), dxy0 = exy, dyy0 = mul(0.5, sub(eyy, exx));
    double gammadot = root(mul(2.0, add(add(mul(dxx0, dxx0), mul(mul(2.0, dxy0), dxy0)),
                                              mul(dyy0, dyy0))));
    double nup_tau, dpxx, dpxy, dpyy;
    if (p_t > c && gf > 0) {
        nup_tau = quot(mul(gf, tau_t), p_t);
        if (nup_tau < 0) nup_tau = 0;
        if (nup_tau > gammadot) nup_tau = gammadot;
        dpxx = mul(mul(r, nup_tau), Npxx);
        dpxy = mul(mul(r, nup_tau), Npxy);
        dpyy = mul(mul(r, nup_tau), Npyy);
    } else {
        nup_tau = 0; dpxx = 0; dpxy = 0; dpyy = 0;
    }
    if (t == 0) {
        nup_tau = 0; dpxx = 0; dpxy = 0; dpyy = 0;
    }
    double exx_e = sub(exx, dpxx), eyy_e = sub(eyy, dpyy);
    dsjxx = mul(mul(dt, cA), add(exx_e, mul(NUMOD, eyy_e)));
    dsjxy = mul(mul(dt, cB), sub(exy, dpxy));
    dsjyy = mul(mul(dt, cA), add(eyy_e, mul(NUMOD, exx_e)));
    dsjxx = sub(dsjxx, jw);
    dsjxy = add(dsjxy, mul(mul(dt, wxy), sub(sxx, syy)));
    dsjyy = add(dsjyy, jw);
    gammap = add(gammap, mul(nup_tau, dt));
    sxx = add(sxx, dsjxx);
    sxy = add(sxy, dsjxy);
    syy = add(syy, dsjyy);
    (void)G;
}

}  // namespace mat
