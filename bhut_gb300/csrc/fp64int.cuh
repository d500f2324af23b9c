// IEEE FP64 products and inverse square roots, correctly rounded, on the
// integer and FP32 pipes.
//
// On GB300 an FP64 warp instruction takes its SM sub-partition about 64
// clocks, and the runtime's square root and division are a dozen of them
// each: the pair loop of form "exact" and of the direct sum spent 2,700 clocks
// on a pair, 29 of its 42 FP64 instructions on products, 1 / sqrt and tests.
// Everything here runs beside the FP64 pipe, which keeps the additions.
//
// The functions are exact by construction, not by an error estimate: a
// product is a 106-bit integer rounded once; a root or a reciprocal is an
// integer candidate from float-float arithmetic, corrected by its remainder,
// which is an exact integer (taken modulo 2^64: the true remainder is far
// below 2^63), and the last step is the definition of round-to-nearest on
// that remainder.  What leaves the normal range belongs to the FP64
// instructions, and callers keep those behind a call: a short fallback in
// line is run under a false predicate, and a predicated FP64 instruction
// occupies the pipe all the same.
//
// BHUT_FP64INT_HOST: the including file supplies the few device intrinsics
// (a check of the same source on the CPU).
#pragma once
#include <cstdint>

#ifndef BHUT_FP64INT_HOST
#include <cuda_runtime.h>
#define BHUT_FN static __device__ __forceinline__
namespace bhut {
namespace fp64int {
// (opaque: tests of the bits would be turned into FP64 comparisons)
BHUT_FN uint64_t bits(double x)
{
    uint64_t b = (uint64_t)__double_as_longlong(x);
    asm("" : "+l"(b));
    return b;
}
BHUT_FN double from_bits(uint64_t b) { return __longlong_as_double((long long)b); }
BHUT_FN uint32_t fbits(float x) { return __float_as_uint(x); }
BHUT_FN float from_fbits(uint32_t b) { return __uint_as_float(b); }
BHUT_FN float fma32(float a, float b, float c) { return __fmaf_rn(a, b, c); }
BHUT_FN float add32(float a, float b) { return __fadd_rn(a, b); }
BHUT_FN float mul32(float a, float b) { return __fmul_rn(a, b); }
BHUT_FN int to_int(float x) { return __float2int_rn(x); }
BHUT_FN float to_float(int x) { return __int2float_rn(x); }
BHUT_FN double sqrt64(double a) { return __dsqrt_rn(a); }
BHUT_FN float rsqrt32(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
#else
namespace bhut {
namespace fp64int {
#endif

constexpr uint64_t kFraction = 0xFFFFFFFFFFFFFull, kOne = 1ull << 52;

// A double taken apart: the mantissa with its leading one at bit 63 (no
// meaning for zero), sign (bit 31) and exponent field.
struct Parts {
    uint64_t m;
    uint32_t sign;
    int e;
    bool zero;
};

BHUT_FN Parts parts(double a)
{
    const uint64_t b = bits(a);
    const uint32_t h = (uint32_t)(b >> 32);
    return Parts{(b << 11) | 0x8000000000000000ull, h & 0x80000000u, (int)((h >> 20) & 0x7ff),
                 ((h << 1) | (uint32_t)b) == 0};
}

// Whether the exponent lies within 2^lo .. 2^hi (or the number is zero).
BHUT_FN bool within(const Parts& a, int lo, int hi)
{
    return a.zero || (unsigned)(a.e - (1023 + lo)) <= (unsigned)(hi - lo);
}

// High word of a b, its last bit set when any lower bit of the product is.
BHUT_FN uint64_t mul_sticky(uint64_t a, uint64_t b)
{
    const uint32_t a0 = (uint32_t)a, a1 = (uint32_t)(a >> 32);
    const uint32_t b0 = (uint32_t)b, b1 = (uint32_t)(b >> 32);
    const uint64_t t = (uint64_t)a0 * b0;
    const uint64_t u = (uint64_t)a1 * b0 + (t >> 32);          // no sum overflows
    const uint64_t v = (uint64_t)a0 * b1 + (uint32_t)u;
    const uint64_t w = (uint64_t)a1 * b1 + (u >> 32) + (v >> 32);
    return w | (((uint32_t)t | (uint32_t)v) != 0);
}

// RN(a b), taken apart (its exponent field may lie outside 1..2046).
BHUT_FN Parts product(const Parts& a, const Parts& b)
{
    uint64_t hi = mul_sticky(a.m, b.m);
    int e = a.e + b.e - 1022;
    if (!(hi >> 63)) { hi += hi; e--; }     // leading one at bit 63
    hi += 0x3ff + ((hi >> 11) & 1);         // nearest at bit 11, ties to even
    if (!(hi >> 63)) { hi = 0x8000000000000000ull; e++; }   // rounded up to 2^64
    return Parts{hi & ~0x7ffull, a.sign ^ b.sign, e, a.zero || b.zero};
}

// RN(a b) as a double (the carry of the rounding runs into the exponent).
BHUT_FN double mul(const Parts& a, const Parts& b)
{
    uint64_t hi = mul_sticky(a.m, b.m);
    int e = a.e + b.e - 1024;
    if (hi >> 63) e++;
    else hi += hi;
    const uint64_t x = hi >> 11;
    const uint32_t up = (((uint32_t)hi & 0x7ff) + ((uint32_t)x & 1) + 0x3ff) >> 11;
    const uint64_t r = (x + up) + ((uint64_t)((uint32_t)e << 20) << 32);
    const bool zero = a.zero || b.zero;
    return from_bits((zero ? 0ull : r) | ((uint64_t)(a.sign ^ b.sign) << 32));
}

// Nearest integer to c, |c| < 2^22, and whether c is so close to a half that
// an error of 2^-12 could change it.
BHUT_FN int nearest(float c, bool& unsure)
{
    const float t = add32(c, 12582912.0f), d = add32(c, -add32(t, -12582912.0f));
    const float off = add32(d < 0.0f ? -d : d, -0.5f);
    unsure = off > -0x1p-11f;
    return (int)fbits(t) - 0x4B400000;
}

// sqrt(x) and 1 / RN(sqrt(x)) for x = X 2^-52 in [1, 4), as integers: m =
// RN(sqrt(x)) in units of 2^-52, v = RN(1 / m) in units of 2^-53.  A
// candidate from float-float arithmetic (within 2^-44) leaves a remainder
// that fits 64 bits; the correction k = remainder / slope is known to 2^-12,
// and only where that does not settle the rounding is the remainder of the
// corrected candidate looked at.
struct Root {
    float y, yl;      // 1 / sqrt(x) to about 2^-45
    uint64_t m;
};

BHUT_FN Root root(uint64_t fraction, int p)   // X = (kOne | fraction) << p
{
    const uint32_t P = (uint32_t)p << 23;
    // x = xh + xl in FP32 (xl to 2^-47: half a step added for the bits cut)
    const float xh = from_fbits(0x3f800000u + P + (uint32_t)(fraction >> 29));
    const float xl = add32(from_fbits(0x34000000u + P + ((uint32_t)(fraction >> 6) & 0x7fffff)),
                           -from_fbits(0x33ffffffu + P));
    Root r;
    // y (1 - A / 2 + 3 A^2 / 8), A = x y^2 - 1: the binomial series of
    // (1 + A)^(-1/2)
    float y = rsqrt32(xh);
    y = y < 0.5f ? 0.5f : (y > 1.0f - 0x1p-24f ? 1.0f - 0x1p-24f : y);
    const float Y = mul32(y, y), Ye = fma32(y, y, -Y);
    const float A = add32(fma32(xh, Y, -1.0f), fma32(xl, Y, mul32(xh, Ye)));
    r.y = y;
    r.yl = mul32(mul32(y, A), fma32(0.375f, A, -0.5f));
    // sqrt(x) = x (y + yl) = sh + sl, sh a 24-bit number in [1, 2)
    float sh = mul32(xh, y);
    sh = sh < 1.0f ? 1.0f : (sh > 2.0f - 0x1p-23f ? 2.0f - 0x1p-23f : sh);
    const float sl = fma32(xh, r.yl, fma32(xl, y, fma32(xh, y, -sh)));
    // candidate m0 in units of 2^-50, remainder t0 in units of 2^-100
    const uint64_t m0 = ((uint64_t)((fbits(sh) & 0x7fffff) | 0x800000) << 27) +
                        (uint64_t)(int64_t)to_int(mul32(sl, 0x1p50f));
    const uint64_t t0 = ((uint64_t)((uint32_t)fraction << p) << 48) - m0 * m0;
    bool unsure;
    const int k = nearest(mul32(to_float((int)(t0 >> 32)), mul32(y, 0x1p-17f)), unsure);
    uint64_t m = (m0 << 2) + (uint64_t)(int64_t)k;
    if (unsure) {
        // X 2^52 = m^2 + t: m is nearest when -m < t <= m
        const int64_t t = (int64_t)((t0 << 4) - (uint64_t)(int64_t)k * ((m0 << 2) + m));
        if (t > (int64_t)m) m++;
        else if (t <= -(int64_t)m) m--;
    }
    r.m = m;
    return r;
}

BHUT_FN uint64_t reciprocal(const Root& r)
{
    const uint64_t r0 = ((uint64_t)((fbits(r.y) & 0x7fffff) | 0x800000) << 27) +
                        (uint64_t)(int64_t)to_int(mul32(r.yl, 0x1p51f));
    const uint64_t u0 = 0ull - r0 * r.m;                 // 2^103 - r0 m, modulo 2^64
    bool unsure;
    const int k = nearest(mul32(to_float((int)(u0 >> 32)), mul32(r.y, 0x1p-18f)), unsure);
    uint64_t v = (r0 << 2) + (uint64_t)(int64_t)k;
    if (unsure) {
        const int64_t u = (int64_t)((u0 << 2) - (uint64_t)(int64_t)k * r.m);   // 2^105 - v m
        if (2 * u > (int64_t)r.m) v++;
        else if (2 * u < -(int64_t)r.m) v--;
    }
    return v;
}

BHUT_FN bool normal_positive(uint64_t b) { return (unsigned)((int)(b >> 52) - 1) < 2046u; }

// RN(sqrt(a)).
BHUT_FN double sqrt(double a)
{
    const uint64_t b = bits(a);
    if (!normal_positive(b)) return sqrt64(a);
    const int e = (int)(b >> 52), p = (e & 1) ^ 1;
    const Root r = root(b & kFraction, p);
    return from_bits(((uint64_t)(1022 + ((e - 1023 - p) >> 1)) << 52) + r.m);
}

// RN(1 / RN(sqrt(a))) of a normal, positive a, taken apart.
BHUT_FN Parts rsqrt(const Parts& a)
{
    const int p = (a.e & 1) ^ 1;
    const Root r = root((a.m >> 11) & kFraction, p);
    const uint64_t v = reciprocal(r);
    const int e = 1022 - ((a.e - 1023 - p) >> 1);
    const bool one = (v >> 53) != 0;          // sqrt is a power of two
    return Parts{one ? 0x8000000000000000ull : v << 11, 0u, e + one, false};
}

}  // namespace fp64int
}  // namespace bhut
