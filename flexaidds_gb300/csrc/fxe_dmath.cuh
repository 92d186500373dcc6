// fxe_dmath.cuh — double-precision quotients and square roots, correctly rounded, with five and four
// FP64 instructions, and conversions and comparisons on the integer units.
//
// GB300's FP64 unit takes one warp instruction per 64 cycles and SM quarter, whatever its active
// lanes (measured: 66 cycles per DFMA of one warp, dependent or not; 16.4 per SM with four or more
// warps; conversions from and to double and comparisons cost the same), and a plain quotient or root
// takes as long as nine of them (146 cycles per SM, measured). Here the reciprocal (or reciprocal
// root) of the operand's significand comes from the single-precision unit — its approximation, then
// one Newton-Raphson step on the operand split in two floats, about 45 bits — and is put together as
// a double with integer arithmetic.
//
// Quotient: one more Newton step in double (two fused multiply-adds) leaves the reciprocal y within half
// a unit and 2^-84 of 1/b, so z0 = a y is within one and a half units in the last place of a / b, and z1 =
// z0 + (a - b z0) y, whose residual is exact, is correctly rounded (after P. W. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990, who asks for the
// correctly rounded reciprocal; y is not that where 1/b itself lies within 2^-84 of a midpoint). For, with
// b in [1, 2): before its rounding z1 is off by (a/b - z0) (b y - 1), and only a quotient beside the
// midpoint of two doubles could round wrongly; there |a/b - z0| is half a unit, |b y - 1| at most
// b (2^-54 + 2^-84), and a/b no nearer to the midpoint than 2^-53 / b units. So b must exceed 2 - 2^-28:
// a divisor whose significand starts with 29 ones falls back to the plain operator. (Of 159,000
// quotients beside midpoints, a third of them by divisors 2 - k 2^-52, three were one unit off when only
// k = 1 fell back.)
//
// Root: g = x (2 h) is within 2^-44 of the root, and g + (x - g g) h within 2^-86 of it before its
// rounding, so the rounded g is the correctly rounded root unless the root lies within 2^-33 units in
// the last place of the midpoint of two doubles. A second correction cannot decide those: it is multiplied
// by the same h, and a root can lie within 2^-54 units of a midpoint. Beside a midpoint the residual
// x - g g is 2 g times half a unit, so its significand is g's (beside_midpoint, an integer test on 20
// bits, one operand in 300,000): those fall back to the plain function.
//
// Both equal the plain operators bit for bit (tests: operands of every kind, and the operands whose
// results lie closest to midpoints); an exponent out of the range the steps need falls back to them
// too. The plain operators sit in functions of their own that are called, so that the short forms do
// not carry them.
#pragma once

#include <cstdint>

namespace fxe {

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// --- comparisons on bit patterns (false when a NaN, of either sign, is involved) -----------------
constexpr long long kInfBits = 0x7ff0000000000000ll;
__device__ __forceinline__ long long bits(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ bool gt0(double x) { return bits(x) > 0 && bits(x) <= kInfBits; }   // x > 0
__device__ __forceinline__ bool lt0(double x) { return gt0(-x); }                               // x < 0
__device__ __forceinline__ bool is0(double x) { return (bits(x) << 1) == 0; }
// a < b and a <= b of values whose sign bit is clear (unsigned: a NaN with the bit set lies above them too)
__device__ __forceinline__ bool lt_nn(double a, double b) {
    const unsigned long long ua = (unsigned long long)bits(a), ub = (unsigned long long)bits(b);
    return ua < ub && ub <= (unsigned long long)kInfBits;
}
__device__ __forceinline__ bool le_nn(double a, double b) {
    const unsigned long long ua = (unsigned long long)bits(a), ub = (unsigned long long)bits(b);
    return ua <= ub && ub <= (unsigned long long)kInfBits;
}

// Biased exponents of operands the short forms take: 2^-350 .. 2^350.
constexpr unsigned kExpLo = 673, kExpSpan = 701;

__device__ __forceinline__ int biased_exp(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// The significand of x as a float in [1, 2), truncated.
__device__ __forceinline__ float top_float(double x) {
    return __uint_as_float(0x3f800000u | ((unsigned)(__double2hiint(x) & 0xfffff) << 3) |
                           ((unsigned)__double2loint(x) >> 29));
}

// (double)x on the integer units (a denormal or special x: the plain conversion).
__device__ __forceinline__ double f2d(float x) {
    const unsigned u = __float_as_uint(x), m = u & 0x7fffffffu;
    double d = __hiloint2double((int)((u & 0x80000000u) | ((m >> 3) + (m ? 0x38000000u : 0u))), (int)(u << 29));
    if (m - 1u < 0x7fffffu || m >= 0x7f800000u) d = (double)x;
    return d;
}

// x as a float, truncated; 0 below the normal range, infinity above it.
__device__ __forceinline__ float d2f_trunc(double x) {
    const int hi = __double2hiint(x);
    const int h = (hi & 0x7fffffff) - 0x38000000;
    unsigned u = __funnelshift_l((unsigned)__double2loint(x), (unsigned)h, 3);
    if (h < 0x100000) u = 0u;
    if (h >= 0x0ff00000) u = 0x7f800000u;
    return __uint_as_float(u | ((unsigned)hi & 0x80000000u));
}

// (r + yl) * 2^k, r in [0.5, 1] and |yl| < 2^-18: the sum as an integer of 2^-62, whose top 53 bits
// complete the exponent field (1021 + k).
__device__ __forceinline__ double join_recip(float r, float yl, int k) {
    // (the approximation may land a step outside [0.5, 1])
    const float rc = fminf(fmaxf(r, 0.5f), 1.0f);
    yl += r - rc;
    const unsigned rb = __float_as_uint(rc);
    const unsigned mant = ((rb & 0x7fffffu) | 0x800000u) << ((rb >> 23) - 126u);   // rc * 2^24
    const long long y62 = ((long long)mant << 38) + ((long long)__float2int_rn(yl * 0x1.0p48f) << 14);
    return __longlong_as_double((y62 >> 9) + ((long long)(1021 + k) << 52));
}

// 1 / |b| to about 45 bits.
__device__ __forceinline__ double recip45(double b) {
    const float bh = top_float(b);
    const float bl = (float)(__double2loint(b) & 0x1fffffff) * 0x1.0p-52f;
    const float r = rcp_approx(bh);
    float e = fmaf(-bh, r, 1.0f);
    e = fmaf(-bl, r, e);
    return join_recip(r, r * fmaf(e, e, e), 1023 - biased_exp(b));
}

// 1 / (2 sqrt(x)) for x > 0 to about 45 bits.
__device__ __forceinline__ double half_rsqrt45(double x) {
    const int ex = (__double2hiint(x) >> 20) - 1023;
    const float sc = (ex & 1) ? 2.0f : 1.0f;
    const float xh = top_float(x) * sc;
    const float xl = (float)(__double2loint(x) & 0x1fffffff) * (sc * 0x1.0p-52f);
    const float r = rsqrt_approx(xh);
    const float r2 = r * r, r2l = fmaf(r, r, -r2);
    float t = fmaf(-xh, r2, 1.0f);
    t = fmaf(-xh, r2l, t);
    t = fmaf(-xl, r2, t);
    return join_recip(r, r * t * fmaf(t, 0.375f, 0.5f), -(ex >> 1) - 1);
}

// a / b; *slow: the plain operator is needed.
__device__ __forceinline__ double div_short(double a, double b, bool* slow) {
    const double ab = fabs(b);
    double y = recip45(b);
    y = __fma_rn(__fma_rn(-ab, y, 1.0), y, y);
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-ab, q, a), y, q);
    if (__double2hiint(b) < 0) q = -q;
    const bool a_ok = (unsigned)(biased_exp(a) - (int)kExpLo) < kExpSpan || (__double2hiint(a) | __double2loint(a)) == 0;   // (-0: the plain operator)
    const bool ones = (((unsigned)__double2hiint(b) | 0xfff00000u) & ((unsigned)__double2loint(b) | 0x00ffffffu)) == 0xffffffffu;
    *slow = !a_ok || (unsigned)(biased_exp(b) - (int)kExpLo) >= kExpSpan || ones;
    return q;
}

// Whether residual r is v times half a unit in the last place of z, both to 20 bits: the half below z (the
// smaller one when z is a power of two) or the half above. hz: z's high word, its sign bit clear.
__device__ __forceinline__ bool beside_midpoint(double r, double v, int hz) {
    const int half = (__double2hiint(v) & 0x7fffffff) + (hz & 0x7ff00000) - (1077 << 20);   // v 2^(e(z) - 54)
    const unsigned k = (unsigned)((__double2hiint(r) & 0x7fffffff) - half + 1);
    return (k & ~(1u << 20)) <= 2u;
}

// sqrt(x); *slow: the plain function is needed.
__device__ __forceinline__ double sqrt_short(double x, bool* slow) {
    const double h = half_rsqrt45(x);
    double g = __dmul_rn(x, __hiloint2double(__double2hiint(h) + (1 << 20), __double2loint(h)));
    g = __fma_rn(__fma_rn(-g, g, x), h, g);
    const int hg = __double2hiint(g);
    // (x - g g = (root - g) 2 g: half a unit of g times 2 g)
    *slow = (unsigned)((__double2hiint(x) >> 20) - (int)kExpLo) >= kExpSpan ||
            beside_midpoint(__fma_rn(-g, g, x), __hiloint2double(hg + (1 << 20), 0), hg);
    return g;
}

static __device__ __noinline__ double plain_div(double a, double b) { return a / b; }
static __device__ __noinline__ double plain_sqrt(double x) { return sqrt(x); }

}  // namespace fxe
