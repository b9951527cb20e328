// lla_pivot_pair.cuh -- one step of the FP32 Cholesky blocks that take two
// columns at a time: the pivots of columns c and c + 1, and what a row needs of
// them, formed by every thread for itself from the two unscaled columns.
//
// Column c + 1 is eliminated first (second()), for the row that is updated and for
// the column it is multiplied with alike, and the trailing entries lose the two
// products of the eliminated columns.  The explicit inverse of the 2 x 2 pivot block,
//     a_ij -= (x0 / d0 - g x1 / d1) t_j + (x1 / d1) u_j,
// is one FMA a column cheaper and as good in exact arithmetic, but its two products
// cancel by a factor sqrt(a_{c+1,c+1} / d1): with nearly collinear neighbouring
// columns (1e-3 apart) its residual was 100 to 700 times that of a column-by-column
// factor, and well-posed matrices (condition 2e7) met a non-positive pivot.  Now the
// two agree, and the entry that is stored as L's is the one the update used.
#pragma once

#include <cuda_runtime.h>

namespace lla {

// Whether a pivot is positive and normal with a normal reciprocal (the approximate
// one flushes subnormal results to zero): 2^-126 <= d < 2^126.  Others take the blocks'
// general forms, which divide by no pivot's reciprocal.
__device__ __forceinline__ bool pivot_pair_takes(float d) { return __float_as_uint(d) - 0x800000u < 0x7e000000u; }

struct PivotPair {
    float d0, r0;  // pivot of column c and its reciprocal
    float d1, r1;  // pivot of column c + 1, after column c
    float g;       // a_{c+1,c} / d0
    // a00 = a_cc, a10 = a_{c+1,c}, a11 = a_{c+1,c+1}
    template <typename Reciprocal>
    __device__ __forceinline__ PivotPair(float a00, float a10, float a11, const Reciprocal &reciprocal) {
        d0 = a00;
        r0 = reciprocal(a00);
        g = a10 * r0;
        d1 = fmaf(-g, a10, a11);
        r1 = reciprocal(d1);
    }
    // a row's entry of column c + 1 after column c, from its entries of both
    __device__ __forceinline__ float second(float x, float y) const { return fmaf(-g, x, y); }
};

// v - s0 t - s1 w: s0, s1 a row's entries over the pivots, t, w a column's, both
// with the second one eliminated.
__device__ __forceinline__ float pivot_pair_apply(float v, float s0, float t, float s1, float w) {
    return fmaf(-s1, w, fmaf(-s0, t, v));
}

}  // namespace lla
