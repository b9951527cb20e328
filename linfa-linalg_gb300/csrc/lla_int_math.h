// lla_int_math.h -- double-precision roots and quotients in integer arithmetic.
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

// ---- correctly rounded quotients by one divisor ------------------------------
//
// a / d with the reciprocal of d's mantissa in fixed point: one high product
// gives the quotient's mantissa with nine or ten bits to spare, below the true
// value by less than two units of the last one.  That decides the rounding (to
// nearest; a quotient of two doubles is never a midpoint) unless the spare bits
// are one short of a half.
struct ImDivisor {
    uint64_t D;   // mantissa of d, 2^52 <= D < 2^53
    uint64_t V;   // floor(2^115 / D)
    int32_t e;    // exponent field of d, sign in bit 11
    int32_t ok;   // d is a normal number
};

__host__ __device__ __forceinline__ ImDivisor im_divisor(double d) {
    const uint64_t b = im_bits(d);
    ImDivisor v;
    v.e = (int32_t)(b >> 52);
    v.ok = im_positive_normal(b & 0x7fffffffffffffffull);
    v.D = (b & 0x000fffffffffffffull) | 0x0010000000000000ull;
    // D 2^-52 in [1, 2) and its reciprocal to 53 bits, then one exact correction:
    // E = 2^115 - V D is below 2^64 in magnitude, so its low 64 bits are E
    const double y = 1.0 / im_double((b & 0x000fffffffffffffull) | 0x3ff0000000000000ull);  // (1/2, 1]
    uint64_t V = (uint64_t)(y * 9223372036854775808.0);  // y 2^63, exact
    if (V > 0x7fffffffffffffffull) V = 0x7fffffffffffffffull;
    int64_t E = (int64_t)(0ull - V * v.D);
    const int64_t k = (int64_t)((double)E * (y * 2.220446049250313e-16));  // E / D, within one of it
    V += (uint64_t)k;
    E -= k * (int64_t)v.D;
    while (E < 0) {
        --V;
        E += (int64_t)v.D;
    }
    while (E >= (int64_t)v.D) {
        ++V;
        E -= (int64_t)v.D;
    }
    v.V = V;
    return v;
}

// a / d; ok says whether it is IEEE division's result (a zero or normal a over a
// normal d with exponents well inside the range, and no undecided rounding).
__host__ __device__ __forceinline__ double im_div(double a, const ImDivisor &d, bool &ok) {
    const uint64_t b = im_bits(a);
    const uint64_t A = (b & 0x000fffffffffffffull) | 0x0010000000000000ull;
    const bool lt = A < d.D, zero = (b << 1) == 0;              // lt: quotient of the mantissas below 1
    const uint64_t hi = im_mulhi(A << 11, d.V);                 // A / D 2^62, less than two above hi
    const uint64_t m = lt ? (hi + 256) >> 9 : (hi + 512) >> 10; // 53 bits, or 2^53
    const int ea = (int)(b >> 52) & 0x7ff, q = ea - (d.e & 0x7ff);
    const uint64_t sign = (b ^ ((uint64_t)(uint32_t)d.e << 52)) & 0x8000000000000000ull;
    const uint64_t e = (uint64_t)(q + 1022 - (lt ? 1 : 0)) << 52;  // biased, minus the leading one of m
    const bool undecided = ((uint32_t)hi & (lt ? 511u : 1023u)) == (lt ? 255u : 511u);
    ok = d.ok && (zero || (ea != 0 && ea != 0x7ff && q > -1020 && q < 1020 && !undecided));
    return im_double(zero ? sign : sign | (e + m));
}

}  // namespace lla
