// lla_oz_digits.h -- the exact-slice digits of a double, as packed BF16 pairs.
// Host and device code: the slicing kernels use these functions, and a host
// test checks them against an independent restatement (digits of
// floor(|a| 2^(56-e)) and the BF16 bits of each signed digit).
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

constexpr int kOzDigits = 8;  // 7-bit digits of a 56-bit magnitude

// The magnitude |a| 2^(56 - e) (|a| < 2^e) as a 56-bit integer, low bits
// truncated (below 2^-56 of the scale), split into its high 28 bits (digits
// 0..3) and low 28 bits (digits 4..7); neg: the sign of a.  Integer operations
// only.  Zero, inf and NaN give 0.
__host__ __device__ __forceinline__ void oz_magnitude(int64_t bits, int e, uint32_t &hi, uint32_t &lo, bool &neg) {
    const int eb = (int)((bits >> 52) & 0x7ff);
    uint64_t mant = (uint64_t)bits & ((1ull << 52) - 1);
    int ea;  // a = mant * 2^ea
    if (eb == 0) {
        ea = -1074;
    } else {
        mant |= 1ull << 52;
        ea = eb - 1075;
    }
    const int shift = ea + 56 - e;  // <= 3 since |a| < 2^e
    uint64_t T = 0;
    if (mant != 0 && eb != 0x7ff) {
        if (shift >= 0)
            T = mant << shift;
        else if (shift > -64)
            T = mant >> (-shift);
    }
    hi = (uint32_t)(T >> 28);
    lo = (uint32_t)(T & 0xfffffffu);
    neg = ((uint64_t)bits >> 63) != 0;
}

// FP32 bits of the signed digit (h >> s) & 127: the digit d is placed in the
// mantissa of 2^23 (exact), and sgn * (2^23 + d) + nsc with (sgn, nsc) = (1,
// -2^23) or (-1, 2^23) is +-d, +0 for d = 0 (an exact zero sum rounds to +0).
// A digit has at most 7 significant bits, so the upper 16 bits are its BF16.
__host__ __device__ __forceinline__ uint32_t oz_digit_f32_bits(uint32_t h, int s, float sgn, float nsc) {
    const uint32_t m = 0x4b000000u | ((h >> s) & 127u);
    float mf, f;
    memcpy(&mf, &m, 4);
#ifdef __CUDA_ARCH__
    f = __fmaf_rn(sgn, mf, nsc);
#else
    f = std::fma(sgn, mf, nsc);
#endif
    uint32_t w;
    memcpy(&w, &f, 4);
    return w;
}

// Two BF16 (the upper halves of two FP32 bit patterns) packed, a in the low half.
__host__ __device__ __forceinline__ uint32_t oz_pack_bf16(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __byte_perm(a, b, 0x7632);
#else
    return (a >> 16) | (b & 0xffff0000u);
#endif
}

// Digits p = 0..7 of four consecutive elements (bits b[0..3], common scale
// exponent e) as BF16: out[p] holds elements 0..3 of plane p, element 0 in the
// lowest 16 bits.
__host__ __device__ __forceinline__ void oz_digits_packed4(const int64_t (&b)[4], int e, uint32_t (&out)[kOzDigits][2]) {
    uint32_t hi[4], lo[4];
    float sgn[4], nsc[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        bool neg;
        oz_magnitude(b[u], e, hi[u], lo[u], neg);
        sgn[u] = neg ? -1.f : 1.f;
        nsc[u] = neg ? 8388608.f : -8388608.f;
    }
#pragma unroll
    for (int p = 0; p < kOzDigits; ++p) {
        const int s = p < 4 ? 7 * (3 - p) : 7 * (7 - p);
        uint32_t f[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) f[u] = oz_digit_f32_bits(p < 4 ? hi[u] : lo[u], s, sgn[u], nsc[u]);
        out[p][0] = oz_pack_bf16(f[0], f[1]);
        out[p][1] = oz_pack_bf16(f[2], f[3]);
    }
}

// ---- balanced 8-bit digits (the trailing updates, lla_fast_chol.cu) ----
//
// An integer of up to 9 bits magnitude 2^7 is exact in BF16, so signed digits
// in [-128, 128] carry 8 bits each: seven of them hold a value rounded to the
// nearest multiple of 2^(e-55), where the truncated 7-bit digits above need
// eight for 56 bits.
constexpr int kOzBal = 7;

// a rounded to the nearest multiple of 2^(e-55) (|a| < 2^e), as that integer
// (|V| <= 2^55); zero for inf and NaN.  Integer operations only.
__host__ __device__ __forceinline__ int64_t oz_fixed55(int64_t bits, int e) {
    const int eb = (int)((bits >> 52) & 0x7ff);
    uint64_t mant = (uint64_t)bits & ((1ull << 52) - 1);
    if (eb != 0) mant |= 1ull << 52;
    const int shift = (eb != 0 ? eb : 1) - 1075 + 55 - e;  // <= 2 since |a| < 2^e
    uint64_t V = 0;
    if (eb != 0x7ff) {
        if (shift >= 0)
            V = mant << shift;
        else if (shift >= -54)
            V = (mant + (1ull << (-shift - 1))) >> (-shift);
    }
    return bits < 0 ? -(int64_t)V : (int64_t)V;
}

// Balanced digits p = 0..6 (most significant first, V = sum_p d_p 256^(6-p)) of
// two values as BF16 pairs, a in the low half of each word.  Adding 128 to every
// digit makes the digits plain bytes (the top one 0..256); a byte in the
// mantissa of 2^23, minus 2^23 + 128, is the signed digit, exact in FP32, and
// its upper 16 bits are its BF16.
__host__ __device__ __forceinline__ void oz_balanced_pair(int64_t va, int64_t vb, uint32_t (&out)[kOzBal]) {
    const uint64_t bias = 0x0080808080808080ull;
    const uint64_t wa = (uint64_t)va + bias, wb = (uint64_t)vb + bias;
#pragma unroll
    for (int p = 0; p < kOzBal; ++p) {
        const int s = 8 * (kOzBal - 1 - p);
        const uint32_t mask = p == 0 ? 0x1ffu : 0xffu;
        const uint32_t ma = 0x4b000000u | ((uint32_t)(wa >> s) & mask), mb = 0x4b000000u | ((uint32_t)(wb >> s) & mask);
        float fa, fb;
        memcpy(&fa, &ma, 4);
        memcpy(&fb, &mb, 4);
        fa -= 8388736.f;
        fb -= 8388736.f;
        uint32_t ba, bb;
        memcpy(&ba, &fa, 4);
        memcpy(&bb, &fb, 4);
        out[p] = oz_pack_bf16(ba, bb);
    }
}

// The same for FP32 values, to the nearest multiple of 2^(e-31) (|V| <= 2^31), in
// four digits.
constexpr int kOzBal32 = 4;
__host__ __device__ __forceinline__ int64_t oz_fixed31(int32_t bits, int e) {
    const int eb = (bits >> 23) & 0xff;
    uint64_t mant = (uint32_t)bits & 0x7fffffu;
    if (eb != 0) mant |= 0x800000u;
    const int shift = (eb != 0 ? eb : 1) - 150 + 31 - e;  // <= 7 since |a| < 2^e
    uint64_t V = 0;
    if (eb != 0xff) {
        if (shift >= 0)
            V = mant << shift;
        else if (shift >= -25)
            V = (mant + (1ull << (-shift - 1))) >> (-shift);
    }
    return bits < 0 ? -(int64_t)V : (int64_t)V;
}
__host__ __device__ __forceinline__ void oz_balanced_pair(int64_t va, int64_t vb, uint32_t (&out)[kOzBal32]) {
    const uint64_t bias = 0x80808080ull;
    const uint64_t wa = (uint64_t)va + bias, wb = (uint64_t)vb + bias;
#pragma unroll
    for (int p = 0; p < kOzBal32; ++p) {
        const int s = 8 * (kOzBal32 - 1 - p);
        const uint32_t mask = p == 0 ? 0x1ffu : 0xffu;
        const uint32_t ma = 0x4b000000u | ((uint32_t)(wa >> s) & mask), mb = 0x4b000000u | ((uint32_t)(wb >> s) & mask);
        float fa, fb;
        memcpy(&fa, &ma, 4);
        memcpy(&fb, &mb, 4);
        fa -= 8388736.f;
        fb -= 8388736.f;
        uint32_t ba, bb;
        memcpy(&ba, &fa, 4);
        memcpy(&bb, &fb, 4);
        out[p] = oz_pack_bf16(ba, bb);
    }
}

// T 2^s outside the normal range; out of line, or the compiler evaluates its FP64
// conversion (64 cycles of the pipe) for every element and selects.
#ifdef __CUDACC__
static __device__ __noinline__ double oz_scaled_rare(int64_t T, int s) { return ldexp((double)T, s); }
#else
static double oz_scaled_rare(int64_t T, int s) { return std::ldexp((double)T, s); }
#endif

// The double nearest to T 2^s, |T| < 2^63 (ties to even): integer operations
// only for results in the normal range.
__host__ __device__ __forceinline__ double oz_scaled_double(int64_t T, int s) {
    const uint64_t u = T < 0 ? 0ull - (uint64_t)T : (uint64_t)T;
#ifdef __CUDA_ARCH__
    const int lz = __clzll((long long)(u | 1));
#else
    const int lz = __builtin_clzll(u | 1);
#endif
    const uint64_t v = u << lz;
    uint64_t m = v >> 11;  // 53 bits, the leading one at bit 52
    const uint32_t rem = (uint32_t)v & 0x7ffu;
    m += rem > 0x400u - ((uint32_t)m & 1) ? 1 : 0;
    const int ex = 63 - lz + s + 1022;  // biased exponent minus one: the leading one of m adds it
    const uint64_t b = ((uint64_t)T & 0x8000000000000000ull) | (((uint64_t)ex << 52) + m);
    double d;
    memcpy(&d, &b, 8);
    if ((uint32_t)ex >= 0x7fdu) {
#if defined(__CUDA_ARCH__) || !defined(__CUDACC__)
        d = oz_scaled_rare(T, s);
#endif
    }
    return T == 0 ? 0.0 : d;
}

// Smallest e with |v| < 2^e for the bit pattern of a finite |v| (0 and
// subnormals: -1022, which holds for all of them).
__host__ __device__ __forceinline__ int oz_bits_exponent(uint64_t abs_bits) {
    const int eb = (int)(abs_bits >> 52);
    return eb == 0 ? -1022 : eb - 1022;
}

}  // namespace lla
