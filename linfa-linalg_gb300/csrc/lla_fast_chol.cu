// lla_fast_chol.cu -- FAST Cholesky, FP64 and FP32: right-looking, lower
// triangle, column-major, with the trailing update on the BF16 tensor cores by
// exact integer digits.
//
// GB300 executes FP64 at about 1.7 operations per clock per SM (measured: one
// FP64 warp instruction occupies its sub-partition for 64 cycles, whatever the
// number of active lanes), 1/64 of the FP32 rate, so n^3/3 flops on the FP64
// pipe take 176 ms at n = 8192 however they are tiled; the FP32 pipe's n^3/3 is
// 1 ms at n = 6001, but its rate needs large register tiles.  Here only the
// O(n^2) parts stay on those pipes:
//   diag   : 64 x 64 diagonal block, one CTA (the update kernel's first, beside
//            the others' tiles);
//   panel  : L21 = A21 L11^-T, 64 columns, by substitution; the finished rows are
//            also cut into balanced 8-bit digits (lla_oz_digits.h; seven for FP64,
//            four for FP32) relative to each row's largest magnitude, exact in
//            BF16;
//   update : A22 -= L21 L21^T with tcgen05 MMAs on the digits.  Every product
//            of digits is an integer of at most 14 bits, a level (sum of the
//            products of equal weight) gathers at most 7 x 128 of them, so the
//            FP32 accumulators hold exact integers (<= 2^24); they are combined
//            in 64-bit integers and subtracted from A22 in its own type: one
//            rounding per entry and 128 columns, where FMAs round once per column.
// Digit products below 2^-56 (FP32: 2^-32) of the row scales are dropped; the
// digits hold each entry to that fraction of its row's largest one.  Panels go in
// pairs: the second one's 64 columns are brought up to date by a narrow update
// with the first panel alone (K = 64), then one update with both (K = 128) covers
// the rest, so the trailing matrix is read and written once per 128 columns.
//
// Measured against updates by FMAs (error against 64 bits the same or lower over
// matrices of that kind; not so for single small entries, include/lla_gb300.h):
// f64 n = 8192 12.3 ms, 220 by FMAs, n = 2048 2.0 and 14.4; f32 n = 6001 2.8 and
// 14.6.  There is no size at which FMAs are faster: one 64 x 64 tile in FP64 takes
// them 70 us on its SM.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "lla_common.cuh"
#include "lla_device.h"
#include "lla_int_math.h"
#include "lla_kernels.h"
#include "lla_oz_mma.cuh"
#include "lla_pivot_pair.cuh"
#include "lla_prof.h"
#include "lla_scratch.h"
#include "lla_tcgen05.cuh"

namespace lla {

constexpr int kFcNb = 64;             // panel width
constexpr int kFcPair = 2 * kFcNb;    // columns per trailing update
constexpr int kFcNonFinite = 1 << 20; // exponent word of a row that holds inf or NaN

// What depends on the element type: digits, their fixed point and exponents, and
// reciprocal roots (of positive normal numbers).
template <typename T>
struct Fc;
template <>
struct Fc<double> {
    static constexpr int kDigits = kOzBal;
    static constexpr int kShift = 62;  // digits of exponents e, f: products in units of 2^(e + f - kShift)
    using Bits = unsigned long long;
    static __device__ __forceinline__ Bits abs_bits(double v) {
        return (Bits)__double_as_longlong(v) & 0x7fffffffffffffffull;
    }
    static __device__ __forceinline__ int exponent(Bits b) {
        return b >= 0x7ff0000000000000ull ? kFcNonFinite : oz_bits_exponent(b);
    }
    static __device__ __forceinline__ int64_t fixed(double v, int e) { return oz_fixed55(__double_as_longlong(v), e); }
    static __device__ __forceinline__ double rsqrt_(double d) { return im_rsqrt(d); }
    static __device__ __forceinline__ bool normal(double d) { return im_positive_normal(im_bits(d)); }
};
template <>
struct Fc<float> {
    static constexpr int kDigits = kOzBal32;
    static constexpr int kShift = 38;
    using Bits = unsigned;
    static __device__ __forceinline__ Bits abs_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
    // (-126 holds for zero and subnormals too)
    static __device__ __forceinline__ int exponent(Bits b) {
        return b >= 0x7f800000u ? kFcNonFinite : max((int)(b >> 23), 0) - 126;
    }
    static __device__ __forceinline__ int64_t fixed(float v, int e) { return oz_fixed31(__float_as_int(v), e); }
    // FP32 approximation and one Newton step
    static __device__ __forceinline__ float rsqrt_(float d) {
        const float y = im_rsqrt_seed(d);
        return fmaf(0.5f * y, fmaf(-d * y, y, 1.f), y);
    }
    static __device__ __forceinline__ bool normal(float d) { return __float_as_uint(d) - 0x800000u < 0x7f000000u; }
};

// Asynchronous copy to shared memory: all of a thread's copies are in flight at once.
template <typename T>
__device__ __forceinline__ void fc_copy(T *dst, const T *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src), "n"(sizeof(T)) : "memory");
}

__device__ __forceinline__ void atomic_min_pos_f64(double *addr, double v) {
    // non-negative doubles order like their bit patterns
    if (v >= 0.0) atomicMin((unsigned long long *)addr, (unsigned long long)__double_as_longlong(v));
}

// Diagonal block [p, p + b), b <= 64, in place; rinv[k] = 1 / L[p+k, p+k] for
// the panel kernel; also min_k pivot_k / A_orig[k, k] for the near-singular
// guard.  Two things bound it: the chain pivot -> reciprocal root -> column ->
// next pivot, and the FP64 pipe of one SM (an instruction takes 64 cycles of
// its sub-partition whatever its active lanes).  Columns go in pairs.  Warp 0
// walks the chain, one pair ahead: it applies pair k to pair k + 1 (two rows a
// lane; one from column 32 on), takes the roots in integer arithmetic and
// scales, without a branch on the way (FP64 comparisons cost 64 cycles as well:
// pivots are tested on their bits, and a bad one redoes the pair).  The warps of
// the other three sub-partitions keep the rest in registers, in patches of 16
// rows x 2 columns (one FP64 instruction per column applied), and hand pair
// k + 2 to warp 0 through shared memory once pair k is in it.  One barrier per
// pair.  31 us a block (one warp for the chain and its columns alike: 160); FP32, where
// fc_diag_quick cannot take it, 13.
constexpr int kFcDiagThreads = 512;
constexpr int kFcPatches = 80, kFcPatchWarps = 12, kFcSlots = 7;

// Patch t, heaviest (rightmost columns) first: row group g, column pair j <= 8 g + 7.
__device__ __forceinline__ void fc_patch(int t, int &g, int &j) {
    if (t < 8) {
        j = 31 - t;
        g = 3;
    } else if (t < 24) {
        j = 23 - (t - 8) / 2;
        g = 3 - (t - 8) % 2;
    } else if (t < 48) {
        j = 15 - (t - 24) / 3;
        g = 3 - (t - 24) % 3;
    } else {
        j = 7 - (t - 48) / 4;
        g = 3 - (t - 48) % 4;
    }
}

// Warp 0: columns c and c + 1 (c even), held in a with all pairs before c - 2
// applied, become columns of L: pair c - 2 applied, pivots, scaling; the pivots
// go to piv, their reciprocal roots to rv.  LOW: c < 32, both halves of the rows
// (lane, lane + 32) take part.  Returns true when a pivot is not positive: its
// column goes to *s_fail and the columns keep what is finished.
template <typename T, bool LOW>
__device__ __forceinline__ bool fc_pivot_pair(T (*a)[kFcNb], T *piv, T *rv, int *s_fail, int c, int lane) {
    T u0 = T(0), v0 = T(0), u1 = a[c][lane + 32], v1 = a[c + 1][lane + 32];
    if (LOW) {
        u0 = a[c][lane];
        v0 = a[c + 1][lane];
    }
    if (c > 0) {
        const T l00 = a[c - 2][c], l01 = a[c - 1][c], l10 = a[c - 2][c + 1], l11 = a[c - 1][c + 1];
        const T x01 = a[c - 2][lane + 32], x11 = a[c - 1][lane + 32];
        if (LOW) {  // the half that holds the pivots first
            const T x00 = a[c - 2][lane], x10 = a[c - 1][lane];
            u0 = fma(-x10, l01, fma(-x00, l00, u0));
            v0 = fma(-x10, l11, fma(-x00, l10, v0));
        }
        u1 = fma(-x11, l01, fma(-x01, l00, u1));
        v1 = fma(-x11, l11, fma(-x01, l10, v1));
    }
    const T su0 = u0, su1 = u1, sv0 = v0, sv1 = v1;
    const T d0 = __shfl_sync(0xffffffffu, LOW ? u0 : u1, c & 31);
    const T y0 = Fc<T>::rsqrt_(d0);
    if (LOW) u0 *= y0;
    u1 *= y0;
    const T l = __shfl_sync(0xffffffffu, LOW ? u0 : u1, (c + 1) & 31);
    if (LOW) v0 = fma(-u0, l, v0);
    v1 = fma(-u1, l, v1);
    const T d1 = __shfl_sync(0xffffffffu, LOW ? v0 : v1, (c + 1) & 31);
    const T y1 = Fc<T>::rsqrt_(d1);
    if (LOW) v0 *= y1;
    v1 *= y1;
    T z0 = y0, z1 = y1;
    int fail = -1;
    if (!Fc<T>::normal(d0) || !Fc<T>::normal(d1)) {
        // not positive (false for NaN, as in the reference), subnormal, inf or NaN: again, with
        // the library's functions
        u0 = su0, u1 = su1, v0 = sv0, v1 = sv1;
        if (d0 <= T(0)) {
            fail = c;
        } else {
            z0 = T(1) / sqrt(d0);
            u0 *= z0;
            u1 *= z0;
            const T l2 = __shfl_sync(0xffffffffu, LOW ? u0 : u1, (c + 1) & 31);
            v0 = fma(-u0, l2, v0);
            v1 = fma(-u1, l2, v1);
            const T e1 = __shfl_sync(0xffffffffu, LOW ? v0 : v1, (c + 1) & 31);
            piv[c + 1] = e1;
            if (e1 <= T(0)) {
                fail = c + 1;
            } else {
                z1 = T(1) / sqrt(e1);
                v0 *= z1;
                v1 *= z1;
            }
        }
        if (lane == 0 && fail >= 0) *s_fail = fail;
    } else {
        piv[c + 1] = d1;
    }
    // (every lane writes the same value)
    piv[c] = d0;
    rv[c] = z0;
    rv[c + 1] = z1;
    if (LOW) {
        a[c][lane] = u0;
        a[c + 1][lane] = v0;
    }
    a[c][lane + 32] = u1;
    a[c + 1][lane + 32] = v1;
    return fail >= 0;
}

// Shared state of a diagonal block's CTA.
template <typename T>
struct FcDiagSmem {
    T a[kFcNb][kFcNb];  // [column][row]
    T piv[kFcNb], rv[kFcNb];
    float pair[3][2][kFcNb];  // FP32: column pairs in turn
    int fail;
};

__device__ __forceinline__ void fc_diag_sync() {
    asm volatile("bar.sync 1, %0;" ::"n"(kFcDiagThreads) : "memory");
}

// FP32 block whose pivots pivot_pair_takes() all: sm.a, sm.piv and sm.rv finished.
// Otherwise sm.fail is set and the block spoilt.  FP32 instructions are short, so
// the chain is exchanges: eight warps hold the block (two rows a lane, eight columns
// a warp), a pair of columns a step goes through shared memory, every thread forms
// its pivots itself (lla_pivot_pair.cuh), and the next pair is brought up to date and
// stored before the columns right of it.  No shuffle, one barrier a pair (of warps
// 0 .. 7).  The factor of n = 6001 takes 2.8 ms, 3.1 with the general form's shuffles.
__device__ __forceinline__ void fc_diag_quick(FcDiagSmem<float> &sm) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = 2 * lane, lc = 8 * warp;
    if (warp >= 8) return;
    float v[8][2];  // column lc + j, row lr + i (above the diagonal: anything)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float2 t = *reinterpret_cast<const float2 *>(&sm.a[lc + j][lr]);
        v[j][0] = t.x, v[j][1] = t.y;
    }
    const auto put = [&](float (*to)[kFcNb], int c, const float (&x)[2], const float (&y)[2]) {
        if (lc == (c & ~7)) {
            *reinterpret_cast<float2 *>(&to[0][lr]) = make_float2(x[0], x[1]);
            *reinterpret_cast<float2 *>(&to[1][lr]) = make_float2(y[0], y[1]);
        }
        asm volatile("bar.sync 2, 256;" ::: "memory");
    };
    const auto reciprocal = [](float d) {  // FP32 approximation and one Newton step
        float r;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
        return fmaf(r, fmaf(-d, r, 1.f), r);
    };
    int b = 0;
    put(sm.pair[0], 0, v[0], v[1]);
#pragma unroll 1
    for (int c8 = 0; c8 < kFcNb; c8 += 8)
#pragma unroll
        for (int j0 = 0; j0 < 8; j0 += 2) {
            const int c = c8 + j0, jn = (j0 + 2) & 7, nb = b == 2 ? 0 : b + 1;
            // (three buffers: a pair's last readers are two barriers before its buffer's reuse)
            const float(*cb)[kFcNb] = sm.pair[b];
            const float2 a0 = *reinterpret_cast<const float2 *>(&cb[0][c]);  // a_cc, a_{c+1,c}
            const float a11 = cb[1][c + 1];
            const float2 x2 = *reinterpret_cast<const float2 *>(&cb[0][lr]);
            const float2 y2 = *reinterpret_cast<const float2 *>(&cb[1][lr]);
            const PivotPair pp(a0.x, a0.y, a11, reciprocal);
            const float d0 = pp.d0, d1 = pp.d1;
            const float x0[2] = {x2.x, x2.y};  // columns c and c + 1, unscaled
            const float x1[2] = {pp.second(x2.x, y2.x), pp.second(x2.y, y2.y)};
            if (lc >= c8) {
                float t[8], u[8], s0[2], s1[2];
#pragma unroll
                for (int h = 0; h < 8; h += 4) {
                    const float4 t4 = *reinterpret_cast<const float4 *>(&cb[0][lc + h]);
                    const float4 u4 = *reinterpret_cast<const float4 *>(&cb[1][lc + h]);
                    t[h] = t4.x, t[h + 1] = t4.y, t[h + 2] = t4.z, t[h + 3] = t4.w;
                    u[h] = u4.x, u[h + 1] = u4.y, u[h + 2] = u4.z, u[h + 3] = u4.w;
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    s0[i] = x0[i] * pp.r0;
                    s1[i] = x1[i] * pp.r1;
                }
                const auto apply = [&](int j) {
                    const float w = pp.second(t[j], u[j]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) v[j][i] = pivot_pair_apply(v[j][i], s0[i], t[j], s1[i], w);
                };
                apply(jn);
                apply(jn + 1);
                put(sm.pair[nb], c + 2, v[jn], v[jn + 1]);  // (c + 2 = 64: nobody's)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j != jn && j != jn + 1) apply(j);
            } else {
                asm volatile("bar.sync 2, 256;" ::: "memory");
            }
            if (warp == 0) {  // the finished pair
                const float q0 = Fc<float>::rsqrt_(d0), q1 = Fc<float>::rsqrt_(d1);
                *reinterpret_cast<float2 *>(&sm.a[c][lr]) = make_float2(x0[0] * q0, x0[1] * q0);
                *reinterpret_cast<float2 *>(&sm.a[c + 1][lr]) = make_float2(x1[0] * q1, x1[1] * q1);
                if (lane == 0) {
                    sm.piv[c] = d0;
                    sm.piv[c + 1] = d1;
                    sm.rv[c] = q0;
                    sm.rv[c + 1] = q1;
                    if (!pivot_pair_takes(d0) || !pivot_pair_takes(d1)) sm.fail = kFcNb;
                }
            }
            b = nb;
        }
}

// By threads 0 .. 511 of a CTA.
template <typename T>
__device__ __forceinline__ void fc_diag_block(FcDiagSmem<T> &sm, T *W, int64_t ld, int64_t p, int b, const T *diag0,
                                              T *rinv, int64_t *info, double *min_ratio) {
    T(*a)[kFcNb] = sm.a;
    T *piv = sm.piv, *rv = sm.rv;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const auto load = [&]() {
#pragma unroll
        for (int e = tid; e < kFcNb * kFcNb; e += kFcDiagThreads) {
            const int r = e % kFcNb, c = e / kFcNb;
            // a short block is padded with the identity
            if (r < b && c <= r)
                fc_copy(&a[c][r], &cm(W, ld, p + r, p + c));
            else
                a[c][r] = T(r == c ? 1 : 0);
        }
        if (tid == 0) sm.fail = -1;
        asm volatile("cp.async.wait_all;" ::: "memory");
        fc_diag_sync();
    };
    load();
    bool done_quick = false;
    if constexpr (sizeof(T) == 4) {
        fc_diag_quick(sm);
        fc_diag_sync();
        done_quick = *(volatile int *)&sm.fail < 0;
        if (!done_quick) {  // (the same for all threads)
            fc_diag_sync();  // every thread has read the verdict
            load();
        }
    }
    const bool upd = (warp & 3) != 0;  // a patch warp (warps 4, 8 and 12 only load and store)
    T acc[kFcSlots];
    int row[kFcSlots], col[kFcSlots];  // col < 0: no patch
    if (upd) {
#pragma unroll
        for (int s = 0; s < kFcSlots; ++s) {
            const int t = warp - 1 - (warp >> 2) + kFcPatchWarps * s;
            int g = 0, j = 0;
            fc_patch(t, g, j);
            row[s] = 16 * g + (lane & 15);
            col[s] = t < kFcPatches ? 2 * j + (lane >> 4) : -1;
            acc[s] = t < kFcPatches ? a[col[s]][row[s]] : T(0);
        }
    }
    bool bad = false;
    if (warp == 0 && !done_quick) bad = fc_pivot_pair<T, true>(a, piv, rv, &sm.fail, 0, lane);
    for (int k = 0; !done_quick; ++k) {
        fc_diag_sync();  // pair k is final
        // A pivot failure of pair k ends the loop for everyone here.  Warp 0 may already have
        // recorded one of pair k + 1 by the time another warp reads the word: that one ends the
        // loop after the next barrier.
        if (warp > 0) bad = (unsigned)*(volatile int *)&sm.fail <= (unsigned)(2 * k + 1);
        if (bad || k == kFcNb / 2 - 1) break;
        if (warp == 0) {
            bad = k < 15 ? fc_pivot_pair<T, true>(a, piv, rv, &sm.fail, 2 * k + 2, lane)
                         : fc_pivot_pair<T, false>(a, piv, rv, &sm.fail, 2 * k + 2, lane);
        } else if (upd) {
#pragma unroll
            for (int s = 0; s < kFcSlots; ++s) {
                if ((col[s] >> 1) < k + 2) break;  // (the same for the whole warp)
                acc[s] = fma(-a[2 * k + 1][row[s]], a[2 * k + 1][col[s]],
                             fma(-a[2 * k][row[s]], a[2 * k][col[s]], acc[s]));
                if ((col[s] >> 1) == k + 2) a[col[s]][row[s]] = acc[s];
            }
        }
    }
    const int fail = bad ? sm.fail : -1;
    const int done = fail >= 0 ? fail : kFcNb;
    if (bad && upd) {  // the columns right of the failing pair, up to date with what was finished
#pragma unroll
        for (int s = 0; s < kFcSlots; ++s)
            if ((col[s] >> 1) > (fail >> 1))
                a[col[s]][row[s]] =
                    (fail & 1) ? fma(-a[fail - 1][row[s]], a[fail - 1][col[s]], acc[s]) : acc[s];
    }
    if (tid < done) {
        rinv[tid] = rv[tid];
        a[tid][tid] = sqrt(piv[tid]);  // exact roots
    }
    if (tid == 0 && fail >= 0) *info = p + fail;
    fc_diag_sync();
    for (int e = tid; e < kFcNb * kFcNb; e += kFcDiagThreads) {
        const int r = e % kFcNb, c = e / kFcNb;
        if (r < b && c <= r) cm(W, ld, p + r, p + c) = a[c][r];
    }
    if (tid < kFcNb && min_ratio) {  // the smallest relative pivot
        double ratio = 1.0e300;
        if (tid < done && tid < b) {
            const double r0 = (double)piv[tid] / (double)diag0[p + tid];
            if (r0 < ratio) ratio = r0;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const double v = __shfl_xor_sync(0xffffffffu, ratio, o);
            if (v < ratio) ratio = v;
        }
        if (lane == 0) atomic_min_pos_f64(min_ratio, ratio);
    }
}

// The first block; the others follow their trailing update in its kernel.
template <typename T>
__global__ void __launch_bounds__(kFcDiagThreads) fc_diag_kernel(T *W, int64_t ld, int64_t p, int b,
                                                                 const T *diag0, T *rinv, int64_t *info,
                                                                 double *min_ratio) {
    __shared__ FcDiagSmem<T> sm;
    pdl_wait();
    pdl_trigger();
    fc_diag_block(sm, W, ld, p, b, diag0, rinv, info, min_ratio);
}

// FP64 panel, between its halves: x[32 + c][r] = sum_k x[k][r] L11[32 + c][k] over
// the 32 finished columns, from byte digits of the 16 rows (wx) and of L11's rows
// (wl, in the space of l11's upper triangle: row 32 + c's at column 32 + c).  By
// 256 threads; ex, el: scale exponents.  Word q of a row and digit: columns q, q +
// 8, q + 16, q + 24; words are swizzled by the row so that a fragment's loads meet
// no bank twice.
__device__ __forceinline__ uint32_t &fc_half_word(uint32_t *row, int i, int d, int q) {
    return row[(d * 8 + q) ^ (4 * (i & 7))];
}

__device__ __forceinline__ int fc_half_digits(uint32_t *row, int i, int q, const double (&v)[4]) {
    unsigned long long mx = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const unsigned long long b = Fc<double>::abs_bits(v[u]);
        mx = b > mx ? b : mx;
    }
#pragma unroll
    for (int o = 1; o < 8; o *= 2) {
        const unsigned long long b = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = b > mx ? b : mx;
    }
    const bool finite = mx < 0x7ff0000000000000ull;
    const int e = finite ? oz_byte_exponent(mx) : kFcNonFinite;
    uint32_t w[kOzBal];
    oz_byte_words(v, e, finite, w);
#pragma unroll
    for (int d = 0; d < kOzBal; ++d) fc_half_word(row, i, d, q) = w[d];
    return e;
}

// Rows that hold inf or NaN have no digits: the FMA chain.
__device__ __noinline__ double fc_half_plain(double v, const double *x, const double *l) {
    for (int k = 0; k < kFcNb / 2; ++k) v = fma(-x[k * (16 + 1)], l[k * kFcNb], v);
    return v;
}

__device__ __forceinline__ void fc_half_product(double (*l11)[kFcNb], double (*x)[16 + 1], uint32_t *wx, int *ex,
                                                int *el) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    {
        const int i = tid >> 3, q = tid & 7;
        const double v[4] = {l11[q][32 + i], l11[q + 8][32 + i], l11[q + 16][32 + i], l11[q + 24][32 + i]};
        const int e = fc_half_digits(reinterpret_cast<uint32_t *>(l11[32 + i]), i, q, v);
        if (q == 0) el[i] = e;
        if (tid < 128) {
            const double u[4] = {x[q][i], x[q + 8][i], x[q + 16][i], x[q + 24][i]};
            const int f = fc_half_digits(wx + i * 64, i, q, u);
            if (q == 0) ex[i] = f;
        }
    }
    __syncthreads();
    if (warp < 4) {  // 8 columns a warp
        float acc[kOzBal][4];
#pragma unroll
        for (int l = 0; l < kOzBal; ++l)
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[l][u] = 0.f;
        uint32_t *lrow = reinterpret_cast<uint32_t *>(l11[32 + 8 * warp + g]);
#pragma unroll
        for (int q = t4; q < 8; q += 4) {
            uint32_t fb[kOzBal][2];
#pragma unroll
            for (int d = 0; d < kOzBal; ++d) oz_byte_digits(fc_half_word(lrow, g, d, q), fb[d][0], fb[d][1]);
#pragma unroll
            for (int d = 0; d < kOzBal; ++d) {
                uint32_t fa[4];
                oz_byte_digits(fc_half_word(wx + g * 64, g, d, q), fa[0], fa[2]);
                oz_byte_digits(fc_half_word(wx + (g + 8) * 64, g, d, q), fa[1], fa[3]);
#pragma unroll
                for (int e = 0; e < kOzBal - d; ++e) oz_mma(acc[d + e], fa, fb[e]);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = g + 8 * (u >> 1), c = 8 * warp + 2 * t4 + (u & 1);
            x[32 + c][r] = oz_scaled_double(oz_byte_sum(acc, u), ex[r] + el[c] - 54);
        }
    }
    __syncthreads();
}

// Panel rows [q, n), q = p + 64: L21 = A21 L11^-T by substitution (multiplying
// by the reciprocal pivots), 16 rows per CTA so that a trailing matrix of 2400
// rows still covers the chip, and the digits of the finished rows.  The rows
// stay in registers as patches of 8 rows x 4 columns, four per warp (warp w: rows
// 8 (w % 2) .., column quads w / 2 + 4 s).  Quads are finished in turn: their two
// owners solve the four columns by shuffles and publish them, one barrier, every
// warp applies them to its quads right of them; the next owners update and solve
// their own quad before the others.  What bounds it is that chain: 16 us a
// panel of FP64 at n = 2048 and 8 of FP32 at n = 6001, against 21 and 13 by pairs of
// columns, with twice the barriers and exchanges.  In FP64 the pipe bounds a panel
// with more than one CTA an SM, so the right half takes the left half's columns from
// the tensor cores instead of by substitution, which halves the FP64 instructions
// (by pairs, n = 8192: 27 us a panel on average, 32 with substitution alone; by quads 24).
// second: the pair of panels' second one -- the rows' first-panel entries are read
// back and the digits of all 128 columns are formed with a common exponent.
constexpr int kFcRows = 16;
constexpr int kFcPanelThreads = 256;

template <typename T>
__global__ void __launch_bounds__(kFcPanelThreads) fc_panel_kernel(T *W, int64_t ld, int64_t n, int64_t p,
                                                                   int second, const T *rinv,
                                                                   __nv_bfloat16 *planes, int64_t plane_stride,
                                                                   int *expo, const int64_t *info) {
    using Bits = typename Fc<T>::Bits;
    constexpr int ND = Fc<T>::kDigits;
    __shared__ T l11[kFcNb][kFcNb];           // [column][row]
    __shared__ T x[kFcNb][kFcRows + 1];    // finished columns, [column][row]
    __shared__ T rv[kFcNb];
    __shared__ Bits s_max[kFcPanelThreads / 16][kFcRows];
    __shared__ int s_e[kFcRows];
    constexpr bool kHalves = sizeof(T) == 8;
    __shared__ uint32_t wx[kHalves ? kFcRows * 64 : 1];
    __shared__ int el[kFcNb / 2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = 8 * (warp & 1) + (lane & 7), c4 = lane >> 3, wq = warp >> 1;
    const int64_t j0 = p + kFcNb + (int64_t)blockIdx.x * kFcRows;
    pdl_wait();
    pdl_trigger();
    if (*(volatile const int64_t *)info >= 0) return;
    // everything the panel reads, in flight at once: L11's lower triangle straight to shared memory
#pragma unroll
    for (int e = tid; e < kFcNb * kFcNb; e += kFcPanelThreads) {
        const int r = e % kFcNb, c = e / kFcNb;
        if (c <= r) fc_copy(&l11[c][r], &cm(W, ld, p + r, p + c));
    }
    T acc[4], first[4];  // first: the pair's first panel
#pragma unroll
    for (int s = 0; s < 4; ++s) acc[s] = j0 + row < n ? cm(W, ld, j0 + row, p + 4 * (wq + 4 * s) + c4) : T(0);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int e = tid + s * kFcPanelThreads, r = e % kFcRows, c = e / kFcRows;
        first[s] = second && j0 + r < n ? cm(W, ld, j0 + r, p - kFcNb + c) : T(0);
    }
    if (tid < kFcNb) rv[tid] = rinv[tid];
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // solves column quad q (this warp's slot value v) and publishes it
    auto solve = [&](int q, T v) {
        const int c = 4 * q;
        const T rc = rv[c + c4], l0 = l11[c][c + c4], l1 = l11[c + 1][c + c4], l2 = l11[c + 2][c + c4];
        // (a lane's v goes on past its own column; nothing reads it there)
        const T u0 = v * rc;
        v = fma(-__shfl_sync(0xffffffffu, u0, lane & 7), l0, v);
        const T u1 = v * rc;
        v = fma(-__shfl_sync(0xffffffffu, u1, 8 + (lane & 7)), l1, v);
        const T u2 = v * rc;
        v = fma(-__shfl_sync(0xffffffffu, u2, 16 + (lane & 7)), l2, v);
        const T u3 = v * rc;
        x[c + c4][row] = c4 & 2 ? (c4 & 1 ? u3 : u2) : (c4 & 1 ? u1 : u0);
    };
    if (wq == 0) solve(0, acc[0]);
    __syncthreads();
#pragma unroll
    for (int s0 = 0; s0 < 4; ++s0) {
        const int send = kHalves && s0 < 2 ? 2 : 4;
        if constexpr (kHalves) {
            if (s0 == 2) {
                fc_half_product(l11, x, wx, s_e, el);
#pragma unroll
                for (int s = 2; s < 4; ++s) {
                    const int c = 4 * (wq + 4 * s) + c4;
                    if (s_e[row] != kFcNonFinite && el[c - 32] != kFcNonFinite)
                        acc[s] -= x[c][row];
                    else
                        acc[s] = fc_half_plain(acc[s], &x[0][row], &l11[0][c]);
                }
                __syncthreads();  // the products have been read
                if (wq == 0) solve(8, acc[2]);
                __syncthreads();
            }
        }
#pragma unroll 1
        for (int w0 = 0; w0 < 4; ++w0) {
            const int j = 4 * s0 + w0;  // quad j is finished: apply it to the quads right of it
            if (j == kFcNb / 4 - 1 || (kHalves && j == kFcNb / 8 - 1)) break;
            T xv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) xv[u] = x[4 * j + u][row];
#pragma unroll
            for (int s = s0; s < send; ++s) {
                const int q = 4 * s + wq;
                if (q <= j) continue;
#pragma unroll
                for (int u = 0; u < 4; ++u) acc[s] = fma(-xv[u], l11[4 * j + u][4 * q + c4], acc[s]);
                if (q == j + 1) solve(q, acc[s]);
            }
            __syncthreads();
        }
    }
    for (int e = tid; e < kFcRows * kFcNb; e += kFcPanelThreads) {
        const int r = e % kFcRows, c = e / kFcRows;
        if (j0 + r < n) cm(W, ld, j0 + r, p + c) = x[c][r];
    }
    // the pair's first panel, in the space of L11
    T(*x1)[kFcRows + 1] = reinterpret_cast<T(*)[kFcRows + 1]>(&l11[0][0]);
    if (second)
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int e = tid + s * kFcPanelThreads;
            x1[e / kFcRows][e % kFcRows] = first[s];
        }
    __syncthreads();
    // row maxima over the pair's columns so far, on the bit patterns
    {
        const int r = tid & 15, g = tid >> 4;  // 16 groups of columns
        Bits mx = 0;
        for (int c = g; c < kFcNb; c += kFcPanelThreads / 16) {
            const Bits v = Fc<T>::abs_bits(x[c][r]);
            mx = v > mx ? v : mx;
            if (second) {
                const Bits u = Fc<T>::abs_bits(x1[c][r]);
                mx = u > mx ? u : mx;
            }
        }
        s_max[g][r] = mx;
    }
    __syncthreads();
    if (tid < kFcRows) {
        Bits mx = 0;
        for (int g = 0; g < kFcPanelThreads / 16; ++g) mx = s_max[g][tid] > mx ? s_max[g][tid] : mx;
        const int e = Fc<T>::exponent(mx);
        s_e[tid] = e;
        if (j0 + tid < n) expo[j0 + tid] = e;
    }
    __syncthreads();
    // digits: four consecutive columns of one row per thread, one 8-byte store a plane
    const int cols = second ? kFcPair : kFcNb;
    for (int e = tid; e < kFcRows * cols / 4; e += kFcPanelThreads) {
        const int k4 = (e % (cols / 4)) * 4, r = e / (cols / 4);
        if (j0 + r >= n) continue;
        const T(*xs)[kFcRows + 1] = second && k4 < kFcNb ? x1 : x;
        const int ks = k4 % kFcNb, ex = s_e[r];
        int64_t v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            v[u] = ex == kFcNonFinite ? 0 : Fc<T>::fixed(xs[ks + u][r], ex);
        uint32_t d0[ND], d1[ND];
        oz_balanced_pair(v[0], v[1], d0);
        oz_balanced_pair(v[2], v[3], d1);
#pragma unroll
        for (int s = 0; s < ND; ++s)
            *reinterpret_cast<uint2 *>(planes + s * plane_stride + (j0 + r) * kFcPair + k4) = make_uint2(d0[s], d1[s]);
    }
}

// ---- trailing update on the tensor cores ------------------------------------

// W[i, j] -= sum_k L[i, p0 + k] L[j, p0 + k], k < 64 kchunks, for i >= j >= q in
// 128 x 64 tiles (row tile I, column tile J <= 2 I + 1; narrow: J = 0 only).
// Persistent CTAs, one per SM, tiles taken in a fixed stride (no CTA waits for
// another).  Per 64-wide K-chunk: the seven digit planes of the 64 column rows
// in one TMA box (double-buffered) and the seven of the 128 rows one after the
// other through a ring; digit plane s of the rows meets planes 0 .. 6 - s of the
// columns in MMAs of N = 64 .. 256 whose results go to consecutive 64-column
// accumulators, one per level s + t (7 x 64 = 448 TMEM columns).  Sixteen warps
// then read the levels, combine them in 64-bit integers, release the tensor
// memory and subtract from W while the next tile's MMAs run.
// Bound by the tensor pipe (28 products), which is 41% busy at n = 8192 because the
// next tile's MMAs wait for the epilogue to have read all levels, and the digit
// planes' L2 traffic (336 KB a tile); the FP64 pipe sees one add per entry.  n = 8192:
// 55 us a panel on average, by FMAs 1403.
constexpr int kFuM = 128, kFuN = 64, kFuK = 64;
constexpr int kFuRing = 6;                         // stages of one row plane
constexpr int kFuATile = kFuM * kFuK * 2;          // 16 KiB
constexpr int kFuBTile = kFuN * kFuK * 2;          // 8 KiB
// All planes of a column tile's chunk (56 KiB for FP64).
template <typename T>
constexpr int kFuBSet = Fc<T>::kDigits *kFuBTile;
template <typename T>
constexpr int kFuSmem = 1024 + kFuRing * kFuATile + 2 * kFuBSet<T> + 256;
constexpr int kFuEpi = 512;                        // 16 epilogue warps (and the next diagonal block's)
static_assert(kFuEpi == kFcDiagThreads && sizeof(FcDiagSmem<double>) <= kFuRing * kFuATile, "");
constexpr int kFuThreads = kFuEpi + 64;            // and the producer's and the MMA issuer's
// Tensor memory: all 512 columns; FP64's seven levels fill 448 of them, FP32's
// four levels leave room for a second set.
constexpr uint32_t kFuTmem = 512;
template <typename T>
constexpr int kFuSets = Fc<T>::kDigits * kFuN * 2 <= (int)kFuTmem ? 2 : 1;

// Entries of rows that hold inf or NaN, which have no digits: the FMA chain on
// the factor itself.
template <typename T>
__device__ __noinline__ T fu_plain_entry(const T *W, int64_t ld, int64_t i, int64_t j, int64_t p0, int kext) {
    T acc = W[i + j * ld];
    for (int k = 0; k < kext; ++k) acc = fma(-W[i + (p0 + k) * ld], W[j + (p0 + k) * ld], acc);
    return acc;
}

__device__ __forceinline__ void fu_tile(int t, int narrow, int &I, int &J) {
    if (narrow) {
        I = t;
        J = 0;
        return;
    }
    // tiles of row I: J = 0 .. 2 I + 1, first index I (I + 1)
    int i = (int)((sqrtf(4.f * (float)t + 1.f) - 1.f) * 0.5f);
    while ((i + 1) * (i + 2) <= t) ++i;
    while (i * (i + 1) > t) --i;
    I = i;
    J = t - i * (i + 1);
}

// W - T 2^s, the product rounded to W's type first.
__device__ __forceinline__ double fu_subtract(double w, long long T, int s) { return w - oz_scaled_double(T, s); }
__device__ __forceinline__ float fu_subtract(float w, long long T, int s) {
    const float t = __ll2float_rn(T);  // 2^t0 with 0 <= t0 <= 47
    // 2^s as a float where it and the product stay normal, scalbnf elsewhere
    const bool fits = s >= -120 && s <= 70;
    return w - (fits ? t * __int_as_float((s + 127) << 23) : scalbnf(t, s));
}

// By the whole CTA, once a bounded wait has run out, instead of the rest of the kernel:
// reports it, lets the copies and MMAs in flight end and frees the tensor memory.
__device__ __forceinline__ void fu_give_up(uint32_t fullA0, uint32_t fullB0, const uint32_t *copied, const uint64_t *drain,
                                        uint32_t tmem, int *err_word, int *sticky) {
    const int tid = threadIdx.x;
    if (tid == 0) {
        atomicCAS(err_word, 0, (int)LLA_ERR_TIMEOUT);
        if (sticky) atomicCAS(sticky, 0, (int)LLA_ERR_TIMEOUT);
    } else if (tid == kFuEpi) {
        ring_drain(fullA0, copied[0], kFuRing);
        ring_drain(fullB0, copied[1], 2);
    } else if (tid == kFuEpi + 32) {
        tc_drain(smem_u32(drain));
    }
    __syncwarp();
    __syncthreads();
    tc_fence_after();
    if (tid < 32)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kFuTmem) : "memory");
}

template <typename T>
__global__ void __launch_bounds__(kFuThreads, 1) fc_update_kernel(
    const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, T *W, int64_t ld,
    int64_t q, int64_t n, int64_t p0, int kchunks, int ntiles, int narrow, const int *__restrict__ expo,
    const T *diag0, T *rinv, int64_t *info, double *min_ratio, int *err_word, int *sticky) {
    constexpr int ND = Fc<T>::kDigits, SETS = kFuSets<T>, BSET = kFuBSet<T>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int s_abort, s_skip;
    __shared__ __align__(8) uint64_t s_drain;
    __shared__ uint32_t s_copied[2];  // planes of rows and of columns that the producer copied
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem;
    uint8_t *sB = smem + kFuRing * kFuATile;
    uint64_t *bars = (uint64_t *)(sB + 2 * BSET);
    uint32_t *tslot = (uint32_t *)(bars + 2 * kFuRing + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t fullA0 = smem_u32(bars), emptyA0 = fullA0 + 8 * kFuRing;
    const uint32_t fullB0 = emptyA0 + 8 * kFuRing, emptyB0 = fullB0 + 16;
    const uint32_t tfull = emptyB0 + 16, tempty = tfull + 16;  // + 8 per set
    if (tid == 0) {
        for (int s = 0; s < kFuRing; ++s) {
            mbar_init(fullA0 + 8 * s, 1);
            mbar_init(emptyA0 + 8 * s, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(fullB0 + 8 * s, 1);
            mbar_init(emptyB0 + 8 * s, 1);
        }
        for (int s = 0; s < SETS; ++s) {
            mbar_init(tfull + 8 * s, 1);
            mbar_init(tempty + 8 * s, kFuEpi);
        }
        mbar_init(smem_u32(&s_drain), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    // the barriers and the tensor memory are set up while the previous kernel ends
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(kFuTmem)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    pdl_wait();
    // One reader decides for the whole CTA (another CTA may report meanwhile; rows from q on are
    // CTA 0's own report on the next block, which stops nobody here).
    if (tid == 0) {
        const int64_t f = *(volatile const int64_t *)info;
        s_skip = (f >= 0 && f < q) || *(volatile const int *)err_word != 0;
    }
    __syncthreads();
    if (s_skip) {
        if (warp == 0)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kFuTmem) : "memory");
        return;
    }
    // CTA 0 takes the first tile alone, the others share the rest
    const int tstep = blockIdx.x ? (int)gridDim.x - 1 : (gridDim.x > 1 ? ntiles : 1);
    // instruction descriptor without N: D F32, A/B BF16, K-major, M = 128
    const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kFuM >> 4) << 24);

    if (warp == kFuEpi / 32) {
        if (lane == 0) {  // TMA producer
            uint32_t ga = 0, gb = 0;
            for (int t = blockIdx.x; t < ntiles && !*(volatile int *)&s_abort; t += tstep) {
                int I, J;
                fu_tile(t, narrow, I, J);
                const int ra = (int)(q + (int64_t)I * kFuM), rb = (int)(q + (int64_t)J * kFuN);
                for (int kc = 0; kc < kchunks && !*(volatile int *)&s_abort; ++kc, ++gb) {
                    const uint32_t xb = gb & 1, use = gb >> 1;
                    if (use > 0 && !mbar_wait(emptyB0 + 8 * xb, (use - 1) & 1, err_word)) {
                        s_abort = 1;
                        break;
                    }
                    mbar_expect_tx(fullB0 + 8 * xb, BSET);
                    tma_load_3d(smem_u32(sB + xb * BSET), &tmB, kc * kFuK, rb, 0, fullB0 + 8 * xb);
                    for (int s = 0; s < ND; ++s, ++ga) {
                        const uint32_t st = ga % kFuRing, round = ga / kFuRing;
                        if (round > 0 && !mbar_wait(emptyA0 + 8 * st, (round - 1) & 1, err_word)) {
                            s_abort = 1;
                            break;
                        }
                        mbar_expect_tx(fullA0 + 8 * st, kFuATile);
                        tma_load_3d(smem_u32(sA + st * kFuATile), &tmA, kc * kFuK, ra, s, fullA0 + 8 * st);
                    }
                }
            }
            s_copied[0] = ga;
            s_copied[1] = gb;
        }
    } else if (warp == kFuEpi / 32 + 1) {
        if (lane == 0) {  // MMA issuer
            uint32_t ga = 0, gb = 0, lt = 0;
            for (int t = blockIdx.x; t < ntiles && !*(volatile int *)&s_abort; t += tstep, ++lt) {
                const uint32_t set = lt % SETS, use = lt / SETS;
                if (use > 0 && !mbar_wait(tempty + 8 * set, (use - 1) & 1, err_word)) {
                    s_abort = 1;
                    break;
                }
                tc_fence_after();
                for (int kc = 0; kc < kchunks && !*(volatile int *)&s_abort; ++kc, ++gb) {
                    const uint32_t xb = gb & 1;
                    if (!mbar_wait(fullB0 + 8 * xb, (gb >> 1) & 1, err_word)) {
                        s_abort = 1;
                        break;
                    }
                    const uint32_t b0 = smem_u32(sB + xb * BSET);
                    for (int s = 0; s < ND; ++s, ++ga) {
                        const uint32_t st = ga % kFuRing;
                        if (!mbar_wait(fullA0 + 8 * st, (ga / kFuRing) & 1, err_word)) {
                            s_abort = 1;
                            break;
                        }
                        tc_fence_after();
                        const uint64_t ad = sw128_desc(smem_u32(sA + st * kFuATile));
                        for (int t0 = 0; t0 < ND - s; t0 += 4) {
                            const int t1 = min(t0 + 4, ND - s);
                            const uint32_t dt = tmem + set * (kFuTmem / SETS) + (uint32_t)((s + t0) * kFuN);
                            const uint32_t idesc = idesc0 | ((uint32_t)((kFuN * (t1 - t0)) >> 3) << 17);
                            const uint64_t bd = sw128_desc(b0 + (uint32_t)(t0 * kFuBTile));
#pragma unroll
                            for (int k = 0; k < kFuK / 16; ++k)  // +32 bytes along K per step
                                tc_mma(dt, ad + 2 * k, bd + 2 * k, idesc, (kc == 0 && s == 0 && k == 0) ? 0u : 1u);
                        }
                        tc_commit(emptyA0 + 8 * st);
                    }
                    if (*(volatile int *)&s_abort) break;
                    tc_commit(emptyB0 + 8 * xb);
                }
                if (*(volatile int *)&s_abort) break;
                tc_commit(tfull + 8 * set);
            }
        }
    } else {  // epilogue: warp w reads lane quarter w % 4, columns 16 (w / 4) .. + 15 of every level
        const int qw = warp & 3, cq = warp >> 2;
        const int r = qw * 32 + lane;
        const uint32_t tcol0 = tmem + ((uint32_t)(qw * 32) << 16) + (uint32_t)(cq * 16);
        uint32_t lt = 0;
        for (int t = blockIdx.x; t < ntiles; t += tstep, ++lt) {
            const uint32_t set = lt % SETS, use = lt / SETS, tcol = tcol0 + set * (kFuTmem / SETS);
            int I, J;
            fu_tile(t, narrow, I, J);
            const int64_t i = q + (int64_t)I * kFuM + r, jb = q + (int64_t)J * kFuN + cq * 16;
            const int nc = i < n ? (int)max((int64_t)0, min((int64_t)16, i - jb + 1)) : 0;  // columns j <= i
            T *wp = W + i + jb * ld;
            // the entries and the columns' exponents (column lane & 15) are fetched before the
            // digits' products are ready
            T w[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) w[c] = c < nc ? wp[c * ld] : T(0);
            const int64_t je = jb + (lane & 15);
            const int ejl = je < n ? expo[je] : 0;
            const int ei = i < n ? expo[i] : 0;
            bool ok = mbar_wait(tfull + 8 * set, use & 1, err_word);
            ok = __all_sync(0xffffffffu, ok) && !*(volatile int *)&s_abort;
            if (!ok) {
                if (lane == 0) s_abort = 1;
                break;
            }
            tc_fence_after();
            // sum_d I_d 2^(8 (ND - 1 - d)).  FP64 needs it less eight bits to fit 64: levels 4-6
            // first, rounded (below the dropped products), then levels 0-3 at 2^16 and up.
            long long sum[16];
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                long long s8[8];
                uint32_t v[8];
                if (ND > 4) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) s8[c] = 128;
#pragma unroll
                    for (int d = 4; d < ND; ++d) {
                        tc_ld8_nowait(tcol + (uint32_t)(d * kFuN + g * 8), v);
                        tc_wait_ld();
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            s8[c] += (long long)__float2int_rn(__uint_as_float(v[c])) * (1 << (8 * (ND - 1 - d)));
                    }
#pragma unroll
                    for (int c = 0; c < 8; ++c) sum[g * 8 + c] = s8[c] >> 8;
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) s8[c] = 0;
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    tc_ld8_nowait(tcol + (uint32_t)(d * kFuN + g * 8), v);
                    tc_wait_ld();
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        s8[c] += (long long)__float2int_rn(__uint_as_float(v[c])) * (1 << (8 * (3 - d)));
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) sum[g * 8 + c] = ND > 4 ? sum[g * 8 + c] + (s8[c] << 16) : s8[c];
            }
            tc_fence_before();
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tempty + 8 * set) : "memory");
            unsigned plain = 0;  // columns to do without digits
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const int ej = __shfl_sync(0xffffffffu, ejl, c);
                const bool nonfinite = ei == kFcNonFinite || ej == kFcNonFinite;
                if (c < nc) {
                    if (nonfinite)
                        plain |= 1u << c;
                    else
                        wp[c * ld] = fu_subtract(w[c], sum[c], ei + ej - Fc<T>::kShift + (ND > 4 ? 8 : 0));
                }
            }
            while (plain) {
                const int c = __ffs(plain) - 1;
                plain &= plain - 1;
                wp[c * ld] = fu_plain_entry(W, ld, i, jb + c, p0, kchunks * kFuK);
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if (s_abort) {
        fu_give_up(fullA0, fullB0, s_copied, &s_drain, tmem, err_word, sticky);
        return;
    }
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kFuTmem) : "memory");
    // The panel kernel may start here and no earlier: its blocks would crowd onto the SMs that this
    // one leaves first (f64 n = 8192: 15.1 ms against 13.6).
    pdl_trigger();
    // The first tile holds the next diagonal block: factored here, in the ring's space (every MMA
    // has read its stages: the epilogue waited for the last one), while the other CTAs go on.  As a
    // kernel of its own between update and panel it leaves the other SMs idle (measured when it went
    // in: f64 n = 8192 13.6 ms, 15.0 as a kernel; n = 2048 2.22, 2.24; f32 n = 6001 3.73, 4.26).
    if (blockIdx.x == 0 && tid < kFcDiagThreads)
        fc_diag_block(*reinterpret_cast<FcDiagSmem<T> *>(smem), W, ld, q, (int)min((int64_t)kFcNb, n - q), diag0, rinv,
                      info, min_ratio);
}

// Saves the input diagonal (for the pivot-ratio guard) and clears the status word.
template <typename T>
__global__ void fc_begin_kernel(const T *W, int64_t ld, int64_t n, T *out, int *err_word) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = cm(W, ld, i, i);
    if (i == 0 && err_word) *err_word = 0;
}

// ---- host side --------------------------------------------------------------

static int fc_encode(PFN_cuTensorMapEncodeTiled_v12000 enc, CUtensorMap *m, void *planes, int64_t n, int digits,
                     int rows, int nplanes) {
    const cuuint32_t estr[3] = {1, 1, 1};
    const cuuint64_t dims[3] = {(cuuint64_t)kFcPair, (cuuint64_t)n, (cuuint64_t)digits};
    const cuuint64_t strides[2] = {(cuuint64_t)kFcPair * 2, (cuuint64_t)n * kFcPair * 2};
    const cuuint32_t box[3] = {(cuuint32_t)kFuK, (cuuint32_t)rows, (cuuint32_t)nplanes};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, planes, dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? 0
               : -1;
}

template <typename T>
int potrf_fast_launch(T *W, int64_t n, int64_t ld, int64_t *d_info, T *diag0, double *min_ratio, int *err_word,
                      int *sticky, cudaStream_t st) {
    constexpr int ND = Fc<T>::kDigits;
    if (allow_dynamic_smem(fc_update_kernel<T>, kFuSmem<T>) != cudaSuccess) return -1;
    const int sms = device_sms();
    PFN_cuTensorMapEncodeTiled_v12000 enc = tma_encoder();
    if (!enc) return -1;
    // digit planes [ND][n][128], row exponents, reciprocal pivots, status word (own copy when
    // the caller passes none)
    const size_t planes_b = (size_t)ND * n * kFcPair * 2, expo_b = ((size_t)n * 4 + 15) / 16 * 16;
    StreamScratch ws(st);
    if (ws.alloc(planes_b + expo_b + kFcNb * 8 + 16) != cudaSuccess) return -1;
    char *base = (char *)ws.get();
    __nv_bfloat16 *planes = (__nv_bfloat16 *)base;
    int *expo = (int *)(base + planes_b);
    T *rinv = (T *)(base + planes_b + expo_b);
    int *own_err = (int *)(base + planes_b + expo_b + kFcNb * 8);
    const int64_t pstride = n * kFcPair;
    int *ew = err_word ? err_word : own_err;
    CUtensorMap tmA, tmB;
    if (fc_encode(enc, &tmA, planes, n, ND, kFuM, 1) || fc_encode(enc, &tmB, planes, n, ND, kFuN, ND)) return -1;
    {
        LaunchScope ls(K_MISC, st);
        fc_begin_kernel<T><<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(W, ld, n, diag0, err_word ? nullptr : own_err);
    }
    const auto panel = [&](int64_t p, int second) {
        const int64_t rest = n - p - kFcNb;
        LaunchScope ls(K_POTRF_FAST_PANEL, st, (double)rest * kFcNb * kFcNb);
        launch_maybe_pdl(true, fc_panel_kernel<T>, dim3((unsigned)ceil_div(rest, kFcRows)), dim3(kFcPanelThreads), 0,
                         st, W, ld, n, p, second, (const T *)rinv, planes, pstride, expo, (const int64_t *)d_info);
    };
    auto update = [&](int64_t q, int64_t p0, int kchunks, int narrow) {
        const int64_t m = n - q, R = ceil_div(m, kFuM);
        // the last row tile may end before its second column tile
        int64_t tiles = narrow ? R : R * (R + 1);
        if (!narrow && ceil_div(m, kFuN) < 2 * R) --tiles;
        const int64_t cols = narrow ? std::min<int64_t>(kFuN, m) : m;
        // algorithmic work: entries of the lower part x columns x 2
        LaunchScope ls(K_POTRF_FAST_UPDATE, st,
                       ((double)m * cols - (double)cols * (cols - 1) / 2) * 2.0 * kchunks * kFuK);
        launch_maybe_pdl(true, fc_update_kernel<T>, dim3((unsigned)std::min<int64_t>(tiles, sms)), dim3(kFuThreads),
                         (size_t)kFuSmem<T>, st, tmA, tmB, W, ld, q, n, p0, kchunks, (int)tiles, narrow,
                         (const int *)expo, (const T *)diag0, rinv, d_info, min_ratio, ew, sticky);
    };
    {
        const int b = (int)std::min<int64_t>(kFcNb, n);
        LaunchScope ls(K_POTRF_FAST_DIAG, st, (double)b * b * b / 3.0);
        launch_maybe_pdl(true, fc_diag_kernel<T>, dim3(1), dim3(kFcDiagThreads), 0, st, W, ld, (int64_t)0, b,
                         (const T *)diag0, rinv, d_info, min_ratio);
    }
    for (int64_t p = 0; p + kFcNb < n; p += kFcPair) {
        panel(p, 0);
        update(p + kFcNb, p, 1, 1);
        if (p + kFcPair >= n) break;
        panel(p + kFcNb, 1);
        update(p + kFcPair, p, 2, 0);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template int potrf_fast_launch<double>(double *, int64_t, int64_t, int64_t *, double *, double *, int *, int *,
                                       cudaStream_t);
template int potrf_fast_launch<float>(float *, int64_t, int64_t, int64_t *, float *, double *, int *, int *,
                                      cudaStream_t);

}  // namespace lla
