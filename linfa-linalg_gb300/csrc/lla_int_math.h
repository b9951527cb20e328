// lla_int_math.h -- double-precision roots and quotients in integer arithmetic,
// single-precision quotients by FMAs.
// Host and device code; a host test checks them against the compiler's.
//
// On GB300 an FP64 instruction takes 64 cycles and occupies its sub-partition
// for all of them; a 64-bit integer multiply takes about 20.  The serial chains
// of the factorisations (pivot -> root -> column) therefore run their Newton
// steps in fixed point from an FP32 seed.
#pragma once

#include <stdint.h>
#include <string.h>

#include <cmath>

#ifndef __CUDACC__  // host-only compilers: the qualifiers vanish
#ifndef __host__
#define __host__
#endif
#ifndef __device__
#define __device__
#endif
#ifndef __forceinline__
#define __forceinline__ inline
#endif
#endif

namespace lla {

__host__ __device__ __forceinline__ uint64_t im_mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

__host__ __device__ __forceinline__ uint64_t im_bits(double d) {
    uint64_t b;
    memcpy(&b, &d, 8);
    return b;
}
__host__ __device__ __forceinline__ double im_double(uint64_t b) {
    double d;
    memcpy(&d, &b, 8);
    return d;
}

// FP32 approximation of 1 / sqrt(m), m in [1, 4), relative error below 2^-21.
__host__ __device__ __forceinline__ float im_rsqrt_seed(float m) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(m));
    return y;
#else
#ifndef IM_SEED_ERROR  // relative error that a test puts on the seed
#define IM_SEED_ERROR 0.0f
#endif
    return (1.0f / std::sqrt(m)) * (1.0f + IM_SEED_ERROR);
#endif
}

// 1 / sqrt(m) as an integer multiple of 2^-61 (error about 2^-60) for
// m = M 2^-62 in [1, 4), mf = m truncated to FP32: FP32 seed y, then one
// third-order step y (1 + r/2 + 3 r^2/8), r = 1 - m y^2 (|r| < 2^-20, the next
// term 5 r^3/16 is below 2^-61).
__host__ __device__ __forceinline__ uint64_t im_rsqrt_q61(uint64_t M, float mf) {
    const float yf = im_rsqrt_seed(mf);  // 1/2 .. 1, or a little outside
    uint32_t yb;
    memcpy(&yb, &yf, 4);
    yb = yb < 0x3f000000u ? 0x3f000000u : (yb > 0x3f7fffffu ? 0x3f7fffffu : yb);  // [1/2, 1)
    const uint32_t Y = (yb & 0x7fffffu) | 0x800000u;          // y 2^24
    const uint64_t P = im_mulhi(M, ((uint64_t)Y * Y) << 15);  // m y^2 2^61
    const int64_t r = (int64_t)((uint64_t)1 << 61) - (int64_t)P;
    const int32_t rh = (int32_t)(r >> 20);
    const int64_t corr = (r >> 1) + ((3 * ((int64_t)rh * rh)) >> 24);
    return ((uint64_t)Y << 37) + (uint64_t)(((int64_t)Y * (corr >> 2)) >> 22);
}

// Whether the bit pattern b is a positive normal number, which the functions
// below take (one integer comparison: FP64 comparisons cost 64 cycles too).
__host__ __device__ __forceinline__ bool im_positive_normal(uint64_t b) {
    return (uint32_t)(b >> 52) - 1u < 0x7feu;  // the sign bit is part of the field
}

// 1 / sqrt(d) to within one unit in the last place, d positive and normal (any
// other d gives a meaningless value).
__host__ __device__ __forceinline__ double im_rsqrt(double d) {
    const uint64_t b = im_bits(d);
    const int eb = (int)(b >> 52);
    const int odd = (eb & 1) ^ 1;                    // d = m 2^(2h), m in [1, 4)
    const int h = (eb - 1023 - odd) >> 1;            // exact
    const uint64_t M = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << (10 + odd);
    const uint32_t fb = ((uint32_t)(127 + odd) << 23) | ((uint32_t)(b >> 29) & 0x7fffffu);
    float mf;
    memcpy(&mf, &fb, 4);
    const uint64_t y = im_rsqrt_q61(M, mf);          // in (2^60, 2^61]
    return im_double(((uint64_t)(1021 - h) << 52) + ((y + 128) >> 8));
}

__host__ __device__ __forceinline__ int64_t im_mulhi_s(int64_t a, int64_t b) {
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return (int64_t)(((__int128)a * b) >> 64);
#endif
}

// ---- correctly rounded quotients by one divisor ------------------------------
//
// 2^115 / D for the divisor's mantissa D as V + F 2^-32: V to 53 bits, F from
// the exact remainder E = 2^115 - V D (below 2^63 in magnitude, so its low 64
// bits are E).  A product with it gives the quotient's mantissa with some 40 bits
// to spare, which decide the rounding (to nearest; a quotient of two doubles is
// never a midpoint) unless they lie within a few units of a half.
struct ImDivisor {
    uint64_t D;   // mantissa of d, 2^52 <= D < 2^53
    uint64_t V;
    int64_t F;    // |F| < 2^43
    int32_t e;    // exponent field of d, sign in bit 11
    int32_t ok;   // d is a normal number
};

// V: 2^115 / D to a relative 2^-53.
__host__ __device__ __forceinline__ void im_reciprocal(ImDivisor &v, uint64_t D, uint64_t V) {
    v.D = D;
    v.V = V;
    v.F = im_mulhi_s((int64_t)(0ull - V * D), (int64_t)V) >> 19;
}

__host__ __device__ __forceinline__ ImDivisor im_divisor(double d) {
    const uint64_t b = im_bits(d);
    ImDivisor v;
    v.e = (int32_t)(b >> 52);
    v.ok = im_positive_normal(b & 0x7fffffffffffffffull);
    const double y = 1.0 / im_double((b & 0x000fffffffffffffull) | 0x3ff0000000000000ull);  // (1/2, 1]
    const uint64_t V = (uint64_t)(y * 9223372036854775808.0);  // y 2^63, exact
    im_reciprocal(v, (b & 0x000fffffffffffffull) | 0x0010000000000000ull, V - (V >> 63));  // below 2^63
    return v;
}

// a / d; ok says whether it is IEEE division's result (a zero or normal a over a
// normal d with exponents well inside the range, and no undecided rounding).
__host__ __device__ __forceinline__ double im_div(double a, const ImDivisor &d, bool &ok) {
    const uint64_t b = im_bits(a);
    const uint64_t An = ((b << 11) & 0x7ffffffffffff800ull) | 0x8000000000000000ull;  // a's mantissa, leading one on top
    const bool lt = An < (d.D << 11), zero = (b << 1) == 0;  // lt: quotient of the mantissas below 1
    // A / D 2^62 = hi . lo, to about 2^-30
    const uint64_t lo0 = An * d.V, hi0 = im_mulhi(An, d.V);
    int64_t G = im_mulhi_s((int64_t)(An >> 1), d.F);         // An F 2^-65
    const uint64_t lo = lo0 + ((uint64_t)G << 33);
    const uint64_t hi = hi0 + (uint64_t)(G >> 31) + (lo < lo0 ? 1 : 0);
    const uint64_t m = lt ? (hi + 256) >> 9 : (hi + 512) >> 10;  // 53 bits, or 2^53
    const int ea = (int)(b >> 52) & 0x7ff, q = ea - (d.e & 0x7ff);
    const uint64_t sign = (b ^ ((uint64_t)(uint32_t)d.e << 52)) & 0x8000000000000000ull;
    const uint64_t e = (uint64_t)(q + 1022 - (lt ? 1 : 0)) << 52;  // biased, minus the leading one of m
    // spare bits and the top of lo, seen from a half
    const int32_t spare = (int32_t)((uint32_t)hi & (lt ? 511u : 1023u)) - (lt ? 256 : 512), top = (int32_t)(lo >> 32) >> 8;
    const bool undecided = (spare == -1 && top == -1) || (spare == 0 && top == 0);
    ok = d.ok && (zero || (ea != 0 && ea != 0x7ff && q > -1020 && q < 1020 && !undecided));
    return im_double(zero ? sign : sign | (e + m));
}

// The same for FP32, where a chain of FMAs is short (4 cycles each; the general
// division's is some 78): the reciprocal rounded to nearest, then Markstein's
// theorem (IBM J. Res. Dev. 34, 1990): a quotient within one unit in the last
// place, its exact remainder and that reciprocal give the rounded quotient.  The
// first of the two corrections brings the quotient within the unit.
struct FloatDivisor {
    float d, y;
    bool ok;
};

// Magnitudes 2^-lo .. 2^hi (a range of bit patterns: false for NaN and infinity).
__host__ __device__ __forceinline__ bool float_within(float v, int lo, int hi) {
    uint32_t b;
    memcpy(&b, &v, 4);
    const uint32_t first = (uint32_t)(127 - lo) << 23, last = (uint32_t)(127 + hi) << 23;
    return (b & 0x7fffffffu) - first <= last - first;
}

__host__ __device__ __forceinline__ FloatDivisor float_divisor(float d) {
    return {d, 1.0f / d, float_within(d, 100, 100)};
}

// a / d ..
__host__ __device__ __forceinline__ float float_div(float a, const FloatDivisor &v) {
    const float q0 = a * v.y;
    const float q1 = fmaf(fmaf(-v.d, q0, a), v.y, q0);
    const float q = fmaf(fmaf(-v.d, q1, a), v.y, q1);
    return a == 0.0f ? q0 : q;  // (the corrections would lose a zero's sign)
}

// .. and whether that is IEEE division's result: a zero, or far enough from the
// ends of the exponent range that the remainders are exact.
__host__ __device__ __forceinline__ bool float_div_ok(float a, float q, const FloatDivisor &v) {
    return v.ok && (a == 0.0f || (float_within(a, 100, 100) && float_within(q, 120, 120)));
}

// sqrt(d), correctly rounded, and the divisor it becomes; d positive and normal.
// The reciprocal root y (2^-60) gives the root to 54 bits or one unit less; the
// exact remainder corrects it, and a root is never a midpoint of two doubles.
// y is also the divisor's reciprocal to 2^-53.
__host__ __device__ __forceinline__ double im_sqrt(double d, ImDivisor &v) {
    const uint64_t b = im_bits(d);
    const int eb = (int)(b >> 52);
    const int odd = (eb & 1) ^ 1;  // d = m 2^(2h), m in [1, 4)
    const int h = (eb - 1023 - odd) >> 1;
    const uint64_t X = (b & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const uint64_t M = X << (10 + odd);
    const uint32_t fb = ((uint32_t)(127 + odd) << 23) | ((uint32_t)(b >> 29) & 0x7fffffu);
    float mf;
    memcpy(&mf, &fb, 4);
    const uint64_t y = im_rsqrt_q61(M, mf);
    // S = floor(sqrt(m) 2^53), or one less
    uint64_t S = (im_mulhi(M, y) - 16) >> 6;
    const int64_t rem = (int64_t)((X << (54 + odd)) - S * S);  // m 2^106 - S^2, modulo 2^64
    S += rem > (int64_t)(2 * S) ? 1 : 0;
    const uint64_t D = (S + 1) >> 1;
    im_reciprocal(v, D, (y << 2) - (y >> 61));  // (below 2^63 for y = 1 too)
    v.e = h + 1023;
    v.ok = 1;
    return im_double(((uint64_t)(h + 1022) << 52) + D);
}

}  // namespace lla
