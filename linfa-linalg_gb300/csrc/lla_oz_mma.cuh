// lla_oz_mma.cuh -- balanced 8-bit digits (lla_oz_digits.h) as bytes in shared
// memory and their products by warp-level FP16 MMAs, for products too small for a
// tcgen05 tile: a digit is exact in FP16, sums of up to 64 products of two exact
// in the FP32 accumulators.
#pragma once

#include "lla_oz_digits.h"

namespace lla {

// D (16 x 8, FP32) += A (16 x 16) B (16 x 8), FP16 operands.
__device__ __forceinline__ void oz_mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Four digits (bytes, biased by 128) as two pairs of FP16: 0x64xx is 1024 + xx.
__device__ __forceinline__ void oz_byte_digits(uint32_t w, uint32_t &lo, uint32_t &hi) {
    const uint32_t a = __byte_perm(w, 0x64646464u, 0x4140), b = __byte_perm(w, 0x64646464u, 0x4342);
    const uint32_t bias = 0x64806480u;  // 1152, 1152
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(lo) : "r"(a), "r"(bias));
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(hi) : "r"(b), "r"(bias));
}

// Scale exponent of values up to the bit pattern mx (finite): one bit of headroom,
// so that the leading digit fits a byte as well.
__device__ __forceinline__ int oz_byte_exponent(uint64_t mx) { return oz_bits_exponent(mx) + 1; }

// Seven digits of four values below 2^(e-1), or of zeros: word d holds byte d of all four.
__device__ __forceinline__ void oz_byte_words(const double (&v)[4], int e, bool finite, uint32_t (&out)[kOzBal]) {
    uint64_t x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
        x[u] = (finite ? (uint64_t)oz_fixed55(__double_as_longlong(v[u]), e) : 0ull) + 0x0080808080808080ull;
    // the four values' bytes 0-3 and 4-6, transposed
    const uint32_t l0 = (uint32_t)x[0], l1 = (uint32_t)x[1], l2 = (uint32_t)x[2], l3 = (uint32_t)x[3];
    const uint32_t h0 = (uint32_t)(x[0] >> 32), h1 = (uint32_t)(x[1] >> 32), h2 = (uint32_t)(x[2] >> 32),
                   h3 = (uint32_t)(x[3] >> 32);
#pragma unroll
    for (int d = 0; d < kOzBal; ++d) {
        const int b = kOzBal - 1 - d;  // byte of the value
        const uint32_t sel = (uint32_t)(b & 3) | (uint32_t)((b & 3) + 4) << 4;
        const uint32_t p01 = b < 4 ? __byte_perm(l0, l1, sel) : __byte_perm(h0, h1, sel);
        const uint32_t p23 = b < 4 ? __byte_perm(l2, l3, sel) : __byte_perm(h2, h3, sel);
        out[d] = __byte_perm(p01, p23, 0x5410);
    }
}

// sum_l acc_l 2^(8 (6 - l)) 2^-8, to the nearest (levels 4-6 are below 2^62 only
// together with that factor), in units of 2^(ei + ej - 54) for scale exponents ei, ej.
__device__ __forceinline__ int64_t oz_byte_sum(const float (&acc)[kOzBal][4], int u) {
    long long lo = 128, hi = 0;
#pragma unroll
    for (int l = 4; l < kOzBal; ++l) lo += (long long)__float2int_rn(acc[l][u]) * (1 << (8 * (6 - l)));
#pragma unroll
    for (int l = 0; l < 4; ++l) hi += (long long)__float2int_rn(acc[l][u]) * (1 << (8 * (3 - l)));
    return hi * 65536 + (lo >> 8);
}

}  // namespace lla
