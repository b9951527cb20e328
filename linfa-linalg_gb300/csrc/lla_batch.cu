// lla_batch.cu -- thousands of independent SPD systems of uneven order in one
// persistent launch.
//
// Layout: the caller packs every system's A_i (n_i x n_i, column-major,
// ld = n_i) into one "A pool" and every B_i (n_i x m_i, ld = n_i) into a "B
// pool" at offsets chosen by the plan.  A plan sorts the systems by
// decreasing cost (n^3/3 + 2 n^2 m) into a device work list; a persistent
// kernel of (CTAs per SM) x (#SMs) blocks takes items from an atomic counter
// (largest first, so the tail is short) and, inside one CTA per system:
//   * factors A_i in place, right-looking with 32-column (FP32) or 16-column
//     (FP64) blocks, the right-hand sides carried along as rows below A_i: the
//     diagonal block is shared out to the CTA's warps, the rows below it are
//     solved against it (a thread, or in short FP64 panels four, per row), and
//     the trailing lower triangle is updated in FP32 register tiles, or for FP64
//     on the tensor cores from 8-bit digits;
//   * solves L^T X = Y, last block first: one warp per right-hand side in the
//     block, one thread per remaining column after it.
// A small system is a chain of latencies, so four CTAs of 128 threads share an SM
// by default; a large FP64 one is bound by the FP64 pipe and the digits' integer
// work.  10,000 systems of n 16-256: f64 5.8 ms, f32 1.2 ms; 3,000 of n 16-64: 0.33
// and 0.13 ms.  (One-warp diagonal blocks with library divisions, FP64 updates on the
// FP64 pipe and two substitution passes: 20.1, 5.4, 1.60 and 0.46 ms.)
// A non-positive pivot stops that system only: info[i] = first failing row
// (-1 when the system solved).  The (CTAs per SM, threads) shape is chosen per
// batch by lla_batch_autotune and cached on disk.
#include <cuda_runtime.h>
#include <sys/stat.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/lla_gb300.h"
#include "lla_autotune.h"
#include "lla_common.cuh"
#include "lla_device.h"
#include "lla_int_math.h"
#include "lla_kernels.h"
#include "lla_oz_mma.cuh"
#include "lla_pivot_pair.cuh"
#include "lla_prof.h"

namespace lla {

constexpr int kBNb = 32;                // block width of the FP32 solves of the refined mode
constexpr int kBMaxN = kBatchMaxN;      // largest order a batch system may have
constexpr int kBMaxRhs = kBatchMaxRhs;  // right-hand sides per system

template <typename T>
__device__ __forceinline__ T shfl(T v, int src) {
    return __shfl_sync(0xffffffffu, v, src);
}

// Block width.  FP32: 32 columns a step.  FP64: 16, because an FP64 instruction
// takes 64 cycles of its sub-partition: half the columns leave half the panel's
// substitution (the rest of it goes to the tensor cores with the update), a
// quarter of the diagonal block, and shared memory and registers for a third CTA.
template <typename T>
constexpr int kBN = sizeof(T) == 4 ? 32 : 16;

// Shared memory of one CTA.
//  dg   : diagonal block, dg[c * kBDs + r] = L[r][c] while factoring (and its
//         transpose in the backward pass), identity-padded;
//  rinv : reciprocals of L's diagonal, all n;
//  rhs  : right-hand sides as extra rows, rhs[k * kBMaxN + i];
//  panel: the finished panel rows: FP32 panel[c * kBPs + r]; FP64 their digits,
//         panel[(d * kBMaxN + r) * 16 + position of k], and expo[r], the rows'
//         exponents.  The right-hand sides' rows follow the matrix rows from the
//         next whole tile on (rhs_row).
constexpr int kBPs = kBMaxN + 4;
constexpr int kBNonFinite = 1 << 20;
template <typename T>
struct BatchSmem {
    static constexpr int kBDs = kBN<T> + 4;  // 16-byte rows in both types
    T dg[kBN<T> * kBDs];
    T rinv[kBMaxN];
    T rhs[kBMaxRhs * kBMaxN];
    T piv[kBN<T>];
    int expo[kBMaxN];
    int fail;
    alignas(16) unsigned char panel[sizeof(T) == 4 ? 4 * kBN<T> * kBPs : kOzBal * kBMaxN * kBN<T>];
};
template <typename T>
__device__ __forceinline__ int rhs_row(int rows) {
    return (rows + kBN<T> - 1) / kBN<T> * kBN<T>;
}
static_assert(kBMaxN - 32 + kBMaxRhs <= kBPs && kBMaxN - 16 + kBMaxRhs <= kBMaxN, "panel rows");

// Asynchronous copy to shared memory: all of a thread's copies are in flight at once.
template <typename T>
__device__ __forceinline__ void batch_copy(T *dst, const T *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(sizeof(T))
                 : "memory");
}

// The same where FP64 has nothing to wait for (the FP64 pipe's work hides it, and the
// refined kernel is 2% slower with it).
__device__ __forceinline__ void batch_fill(float *dst, const float *src) { batch_copy(dst, src); }
__device__ __forceinline__ void batch_fill(double *dst, const double *src) { *dst = *src; }

// 1 / sqrt(d), d positive and normal: FP32 approximation and one Newton step;
// FP64 in fixed point (lla_int_math.h).
__device__ __forceinline__ float batch_rsqrt(float d) {
    const float y = im_rsqrt_seed(d);
    return fmaf(0.5f * y, fmaf(-d * y, y, 1.f), y);
}
__device__ __forceinline__ double batch_rsqrt(double d) { return im_rsqrt(d); }
__device__ __forceinline__ bool batch_normal(float d) { return __float_as_uint(d) - 0x800000u < 0x7f000000u; }
__device__ __forceinline__ bool batch_normal(double d) { return im_positive_normal(im_bits(d)); }

// Factors the identity-padded diagonal block in sm.dg; sm.rinv[kb ..] receives
// the reciprocal pivots, the block L with its exact roots.  sm.fail: failing row.
// Warp 0 walks the pivots, a pair of columns at a time and one pair ahead, and the
// warps of the other sub-partitions apply the finished pairs to the rest in
// patches of 16 rows x 2 columns.
template <typename T>
__device__ void batch_diag(BatchSmem<T> &sm, int kb) {
    constexpr int NB = kBN<T>, DS = BatchSmem<T>::kBDs, NP = NB / 2;
    constexpr int kPatches = NB == 32 ? 24 : 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & (NB - 1);  // (FP64: both half-warps do the same)
    T *a = sm.dg;
    auto pivots = [&](int c) {
        T u = a[c * DS + lane], v = a[(c + 1) * DS + lane];
        if (c > 0) {
            const T *x0 = a + (c - 2) * DS, *x1 = a + (c - 1) * DS;
            u = fma(-x1[lane], x1[c], fma(-x0[lane], x0[c], u));
            v = fma(-x1[lane], x1[c + 1], fma(-x0[lane], x0[c + 1], v));
        }
        const T su = u, sv = v;
        const T d0 = shfl(u, c);
        T y0 = batch_rsqrt(d0);
        u *= y0;
        v = fma(-u, shfl(u, c + 1), v);
        T d1 = shfl(v, c + 1);
        T y1 = batch_rsqrt(d1);
        v *= y1;
        // not positive (NaN does not fail, as in the reference: `d <= 0`), or special
        if (!batch_normal(d0) || !batch_normal(d1)) {
            int fail = d0 <= T(0) ? c : -1;
            y0 = T(1) / sqrt(d0);
            u = su * y0;
            v = fma(-u, shfl(u, c + 1), sv);
            d1 = shfl(v, c + 1);
            if (d1 <= T(0) && fail < 0) fail = c + 1;
            y1 = T(1) / sqrt(d1);
            v *= y1;
            if (tid == 0 && fail >= 0 && sm.fail < 0) sm.fail = kb + fail;
        }
        sm.piv[c] = d0;  // (every lane writes the same value)
        sm.piv[c + 1] = d1;
        sm.rinv[kb + c] = y0;
        sm.rinv[kb + c + 1] = y1;
        __syncwarp();
        a[c * DS + lane] = u;
        a[(c + 1) * DS + lane] = v;
    };
    if (warp == 0) pivots(0);
    const int npw = (blockDim.x >> 7) * 3, pw = warp - 1 - (warp >> 2);
    for (int k = 0; k < NP - 1; ++k) {
        __syncthreads();  // pair k is final
        if (warp == 0) {
            pivots(2 * k + 2);
        } else if (warp & 3) {
            const T *x0 = a + 2 * k * DS, *x1 = x0 + DS;
            for (int t = pw; t < kPatches; t += npw) {  // rightmost pairs first
                const int j = t < 8 ? NP - 1 - t : 7 - (t - 8) / 2, g = NB == 16 ? 0 : (t < 8 ? 1 : 1 - (t & 1));
                if (j < k + 2) break;
                const int r = 16 * g + (tid & 15), c = 2 * j + ((tid >> 4) & 1);
                a[c * DS + r] = fma(-x1[r], x1[c], fma(-x0[r], x0[c], a[c * DS + r]));
            }
        }
    }
    __syncthreads();
    if (tid < NB) a[tid * DS + tid] = sqrt(sm.piv[tid]);
    __syncthreads();
}

// FP32, pivot_pair_takes() every pivot (false otherwise, the block spoilt): four
// warps hold the block, 2 rows x 4 columns a thread.  Two columns a round go through
// shared memory (the panel's space), every thread forms their pivots itself
// (lla_pivot_pair.cuh), and the next pair is brought up to date and stored before the
// columns right of it: one exchange and no shuffle on a pair's chain (10,000 systems
// of n 16-256: 1.12 ms in the kernel, 1.23 with batch_diag).
__device__ bool batch_diag_quick(BatchSmem<float> &sm, int kb) {
    constexpr int DS = BatchSmem<float>::kBDs;
    const int tid = threadIdx.x;
    float *a = sm.dg;
    bool ok = true;
    if (tid < 128) {
        const int lr = 2 * (tid & 15), lc = 4 * (tid >> 4);
        float v[4][2];  // column lc + j, row lr + i (above the diagonal: anything)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 t = *reinterpret_cast<const float2 *>(&a[(lc + j) * DS + lr]);
            v[j][0] = t.x, v[j][1] = t.y;
        }
        float *const bufs = reinterpret_cast<float *>(sm.panel);  // three pairs of columns
        float *cb = bufs;
        const auto put = [&](float *to, int c, const float (&x)[2], const float (&y)[2]) {
            if (lc == (c & ~3)) {
                *reinterpret_cast<float2 *>(to + lr) = make_float2(x[0], x[1]);
                *reinterpret_cast<float2 *>(to + 32 + lr) = make_float2(y[0], y[1]);
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
        };
        const auto reciprocal = [](float d) {
            float r;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
            return fmaf(r, fmaf(-d, r, 1.f), r);
        };
        put(cb, 0, v[0], v[1]);
#pragma unroll 1
        for (int c4 = 0; c4 < 32; c4 += 4)
#pragma unroll
            for (int j0 = 0; j0 < 4; j0 += 2) {
                const int c = c4 + j0, jn = (j0 + 2) & 3;
                float *nb = cb == bufs + 128 ? bufs : cb + 64;
                const float2 a0 = *reinterpret_cast<const float2 *>(cb + c);  // a_cc, a_{c+1,c}
                const float a11 = cb[32 + c + 1];
                const float2 x2 = *reinterpret_cast<const float2 *>(cb + lr);
                const float2 y2 = *reinterpret_cast<const float2 *>(cb + 32 + lr);
                const float4 t4 = *reinterpret_cast<const float4 *>(cb + lc);
                const float4 u4 = *reinterpret_cast<const float4 *>(cb + 32 + lc);
                const float t[4] = {t4.x, t4.y, t4.z, t4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
                const PivotPair pp(a0.x, a0.y, a11, reciprocal);
                const float d0 = pp.d0, d1 = pp.d1;
                const float x0[2] = {x2.x, x2.y};  // columns c and c + 1, unscaled
                const float x1[2] = {pp.second(x2.x, y2.x), pp.second(x2.y, y2.y)};
                const float s0[2] = {x0[0] * pp.r0, x0[1] * pp.r0}, s1[2] = {x1[0] * pp.r1, x1[1] * pp.r1};
                const auto apply = [&](int j) {
                    const float w = pp.second(t[j], u[j]);
#pragma unroll
                    for (int i = 0; i < 2; ++i) v[j][i] = pivot_pair_apply(v[j][i], s0[i], t[j], s1[i], w);
                };
                apply(jn);
                apply(jn + 1);
                put(nb, c + 2, v[jn], v[jn + 1]);  // (c + 2 = 32: nobody's)
                apply(j0);
                apply(j0 + 1);
                ok = ok && pivot_pair_takes(d0) && pivot_pair_takes(d1);
                if (tid < 32) {  // the finished pair, a column for each half of the warp
                    const bool second = tid & 16;
                    const float y = batch_rsqrt(second ? d1 : d0);
                    *reinterpret_cast<float2 *>(&a[(c + (second ? 1 : 0)) * DS + lr]) =
                        make_float2((second ? x1[0] : x0[0]) * y, (second ? x1[1] : x0[1]) * y);
                    if ((tid & 15) == 0) {
                        sm.rinv[kb + c + (second ? 1 : 0)] = y;
                        sm.piv[c + (second ? 1 : 0)] = second ? d1 : d0;
                    }
                }
                cb = nb;
            }
    }
    if (!__syncthreads_and(ok)) return false;
    if (tid < 32) a[tid * DS + tid] = sqrt(sm.piv[tid]);
    __syncthreads();
    return true;
}

// Trailing update of the lower triangle of the rows q + i, i < rows, and of the
// right-hand sides' rows, from the panel.  FP32: warp tiles of 32 x 32, a thread 4
// rows (stride 8) x 8 columns.
template <bool EDGE>
__device__ __forceinline__ void batch_tile(const float *P, float *Aq, int n, int i0, int j0, int rows) {
    float acc[4][8];
#pragma unroll
    for (int w = 0; w < 8; ++w)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            acc[u][w] = !EDGE || (i0 + 8 * u < rows && j0 + w <= i0 + 8 * u) ? Aq[8 * u + w * n] : 0.f;
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
        float xr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) xr[u] = P[k * kBPs + i0 + 8 * u];
        const float4 c0 = *reinterpret_cast<const float4 *>(P + k * kBPs + j0);
        const float4 c1 = *reinterpret_cast<const float4 *>(P + k * kBPs + j0 + 4);
        const float xc[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int w = 0; w < 8; ++w) acc[u][w] = fmaf(-xr[u], xc[w], acc[u][w]);
    }
#pragma unroll
    for (int w = 0; w < 8; ++w)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (!EDGE || (i0 + 8 * u < rows && j0 + w <= i0 + 8 * u)) Aq[8 * u + w * n] = acc[u][w];
}

__device__ void batch_update(BatchSmem<float> &sm, float *A, int n, int q, int kb, int rows, int m) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const float *P = reinterpret_cast<const float *>(sm.panel);
    const int R = (rows + 31) / 32, lr = lane & 7, lc = (lane >> 3) * 8;
    int I = 0, J = warp;  // lower tiles, row by row
    for (;;) {
        while (J > I) {
            J -= I + 1;
            ++I;
        }
        if (I >= R) break;
        const int i0 = 32 * I + lr, j0 = 32 * J + lc;
        float *Aq = A + q + i0 + (int64_t)(q + j0) * n;
        if (J < I && 32 * I + 32 <= rows)
            batch_tile<false>(P, Aq, n, i0, j0, rows);
        else
            batch_tile<true>(P, Aq, n, i0, j0, rows);
        J += nw;
    }
    const int b0 = rhs_row<float>(rows);
    for (int j = threadIdx.x; j < rows; j += blockDim.x) {
        float x[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) x[c] = P[c * kBPs + j];
        for (int k = 0; k < m; ++k) {
            float s = sm.rhs[k * kBMaxN + q + j];
#pragma unroll
            for (int c = 0; c < 32; ++c) s = fmaf(-P[c * kBPs + b0 + k], x[c], s);
            sm.rhs[k * kBMaxN + q + j] = s;
        }
    }
    __syncthreads();
}

// FP64: the product of the 16 panel columns on the tensor cores, from seven
// balanced 8-bit digits per entry (exact in FP16, their products' sums exact in
// the FP32 accumulators), one 64-bit integer per entry and one FP64 subtraction,
// where FMAs would spend 16 FP64 instructions per entry (lla_fast_chol.cu has the
// scheme and its error).  Warp tiles of 16 x 8; the digits' k order is permuted
// alike in both operands so that a thread's four are one word.
__device__ void batch_update(BatchSmem<double> &sm, double *A, int n, int q, int kb, int rows, int m) {
    constexpr int NB = 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int R = (rows + 15) / 16, C = (rows + 7) / 8;  // (row R: the right-hand sides)
    int I = 0, J = warp;                                  // tiles of row I: J <= 2 I + 1, J < C
    for (;;) {
        for (int w = min(2 * I + 2, C); I <= R && J >= w; w = min(2 * I + 2, C)) {
            J -= w;
            ++I;
        }
        if (I > R) break;
        const bool isb = I == R;
        // this thread's entries, fetched before the products
        double *wp[4], w[4];
        int use = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = 16 * I + g + 8 * (u >> 1), j = 8 * J + 2 * t4 + (u & 1);
            const bool in = j < rows && (isb ? i - 16 * R < m : i < rows && j <= i);
            wp[u] = isb ? &sm.rhs[(in ? i - 16 * R : 0) * kBMaxN + q + (in ? j : 0)]
                        : &A[in ? (q + i) + (int64_t)(q + j) * n : 0];
            w[u] = in ? *wp[u] : 0.0;
            use |= in ? 1 << u : 0;
        }
        float acc[kOzBal][4];
#pragma unroll
        for (int l = 0; l < kOzBal; ++l)
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[l][u] = 0.f;
        uint32_t fb[kOzBal][2];
#pragma unroll
        for (int d = 0; d < kOzBal; ++d)
            oz_byte_digits(*reinterpret_cast<const uint32_t *>(sm.panel + (d * kBMaxN + 8 * J + g) * NB + 4 * t4), fb[d][0],
                         fb[d][1]);
#pragma unroll
        for (int d = 0; d < kOzBal; ++d) {
            uint32_t fa[4];
            const unsigned char *pa = sm.panel + (d * kBMaxN + 16 * I + g) * NB + 4 * t4;
            oz_byte_digits(*reinterpret_cast<const uint32_t *>(pa), fa[0], fa[2]);
            oz_byte_digits(*reinterpret_cast<const uint32_t *>(pa + 8 * NB), fa[1], fa[3]);
#pragma unroll
            for (int e = 0; e < kOzBal - d; ++e) oz_mma(acc[d + e], fa, fb[e]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int ei = sm.expo[16 * I + g + 8 * (u >> 1)], ej = sm.expo[8 * J + 2 * t4 + (u & 1)];
            const int64_t sum = oz_byte_sum(acc, u);
            if (use >> u & 1) {
                if (ei != kBNonFinite && ej != kBNonFinite) {
                    *wp[u] = w[u] - oz_scaled_double(sum, ei + ej - 54);
                } else {  // no digits: the FMA chain on the factor itself
                    const int i = 16 * I + g + 8 * (u >> 1), j = 8 * J + 2 * t4 + (u & 1);
                    double s = w[u];
                    for (int k = 0; k < NB; ++k)
                        s = fma(-(isb ? sm.rhs[(i - 16 * R) * kBMaxN + kb + k] : A[(q + i) + (int64_t)(kb + k) * n]),
                                A[(q + j) + (int64_t)(kb + k) * n], s);
                    *wp[u] = s;
                }
            }
        }
        J += nw;
    }
    __syncthreads();
}

// Word t of the digits of panel row rr: columns t, t + 4, t + 8, t + 12.
__device__ __forceinline__ void batch_keep_word(BatchSmem<double> &sm, int rr, int t, const double (&w)[4], int e) {
    uint32_t word[kOzBal];
    oz_byte_words(w, e, e != kBNonFinite, word);
#pragma unroll
    for (int d = 0; d < kOzBal; ++d) *reinterpret_cast<uint32_t *>(sm.panel + (d * kBMaxN + rr) * 16 + 4 * t) = word[d];
}

// Keeps a finished panel row (row rr of the panel) for the update.
__device__ __forceinline__ void batch_keep_row(BatchSmem<float> &sm, int rr, const float (&v)[32]) {
    float *P = reinterpret_cast<float *>(sm.panel);
#pragma unroll
    for (int c = 0; c < 32; ++c) P[c * kBPs + rr] = v[c];
}
__device__ __forceinline__ void batch_keep_row(BatchSmem<double> &sm, int rr, const double (&v)[16]) {
    uint64_t mx = 0;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const uint64_t b = im_bits(v[c]) & 0x7fffffffffffffffull;
        mx = b > mx ? b : mx;
    }
    const int e = mx < 0x7ff0000000000000ull ? oz_byte_exponent(mx) : kBNonFinite;
    sm.expo[rr] = e;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const double w[4] = {v[t], v[t + 4], v[t + 8], v[t + 12]};
        batch_keep_word(sm, rr, t, w, e);
    }
}

// FP64 panel of at most blockDim / 4 rows: four threads a row (eight rows a warp),
// thread t of a row its columns t, t + 4, t + 8, t + 12, so that a short panel
// uses every sub-partition's FP64 pipe and a row's digits are formed four ways.
__device__ void batch_panel_split(double *A, int n, int kb, int bs, int q, int rows, int m, BatchSmem<double> &sm) {
    constexpr int DS = BatchSmem<double>::kBDs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r8 = lane & 7, t = lane >> 3;
    const int rr = warp * 8 + r8;
    if (warp * 8 >= rows + m) return;  // (uniform for the warp)
    const bool in = rr < rows + m, isb = rr >= rows;
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int c = 4 * u + t;
        v[u] = in && c < bs ? (isb ? sm.rhs[(rr - rows) * kBMaxN + kb + c] : A[(q + rr) + (int64_t)(kb + c) * n]) : 0.0;
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const double x = shfl(v[c >> 2] * sm.rinv[kb + c], (c & 3) * 8 + r8);
        if (t == (c & 3)) v[c >> 2] = x;
#pragma unroll
        for (int u = c >> 2; u < 4; ++u) {
            const double w = fma(-x, sm.dg[c * DS + 4 * u + t], v[u]);
            if (4 * u + t > c) v[u] = w;
        }
    }
    if (in) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = 4 * u + t;
            if (c < bs) {
                if (isb)
                    sm.rhs[(rr - rows) * kBMaxN + kb + c] = v[u];
                else
                    A[(q + rr) + (int64_t)(kb + c) * n] = v[u];
            }
        }
    }
    if (rows == 0) return;
    uint64_t mx = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const uint64_t b = im_bits(v[u]) & 0x7fffffffffffffffull;
        mx = b > mx ? b : mx;
    }
#pragma unroll
    for (int o = 8; o < 32; o *= 2) {
        const uint64_t b = __shfl_xor_sync(0xffffffffu, (unsigned long long)mx, o);
        mx = b > mx ? b : mx;
    }
    const int e = mx < 0x7ff0000000000000ull ? oz_byte_exponent(mx) : kBNonFinite;
    if (in) {
        const int p = isb ? rhs_row<double>(rows) + rr - rows : rr;
        if (t == 0) sm.expo[p] = e;
        batch_keep_word(sm, p, t, v, e);
    }
}

// Factor of one system by the whole CTA: A (n x n, column-major, ld = n) in
// place (L in the lower triangle), right-looking; the m right-hand sides in
// sm.rhs are carried along as rows below A, which makes them L^-1 B.  Returns the
// first failing row (non-positive pivot) or -1; every thread returns the same
// value.
template <typename T>
__device__ int batch_factor(T *A, int n, int m, BatchSmem<T> &sm) {
    constexpr int NB = kBN<T>, DS = BatchSmem<T>::kBDs;
    const int tid = threadIdx.x, nthr = blockDim.x;
    if (tid == 0) sm.fail = -1;
    __syncthreads();
    for (int kb = 0; kb < n; kb += NB) {
        const int bs = min(NB, n - kb), q = kb + bs, rows = n - q;
        for (int e = tid; e < NB * NB; e += nthr) {
            const int r = e % NB, c = e / NB;
            if (r < bs && c <= r)
                batch_copy(&sm.dg[c * DS + r], &A[(kb + r) + (int64_t)(kb + c) * n]);
            else
                sm.dg[c * DS + r] = T(r == c ? 1 : 0);
        }
        // the rows below the block, one a thread, fetched while the block is factored
        const int total = rows + m;
        T v[NB];
        auto fetch = [&](int rr) {
#pragma unroll
            for (int c = 0; c < NB; ++c)
                v[c] = c < bs ? (rr < rows ? A[(q + rr) + (int64_t)(kb + c) * n] : sm.rhs[(rr - rows) * kBMaxN + kb + c])
                              : T(0);
        };
        const bool split = sizeof(T) == 8 && 4 * total <= nthr;
        if (tid < total && !split) fetch(tid);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if constexpr (sizeof(T) == 4) {
            if (!batch_diag_quick(sm, kb)) {
                for (int e = tid; e < NB * NB; e += nthr) {
                    const int r = e % NB, c = e / NB;
                    sm.dg[c * DS + r] = (r < bs && c <= r) ? A[(kb + r) + (int64_t)(kb + c) * n] : T(r == c ? 1 : 0);
                }
                __syncthreads();
                batch_diag<T>(sm, kb);
            }
        } else {
            batch_diag<T>(sm, kb);
        }
        if (sm.fail >= 0) break;
        for (int e = tid; e < NB * NB; e += nthr) {
            const int r = e % NB, c = e / NB;
            if (r < bs && c <= r) A[(kb + r) + (int64_t)(kb + c) * n] = sm.dg[c * DS + r];
        }
        if constexpr (sizeof(T) == 8) {
            if (split) batch_panel_split(A, n, kb, bs, q, rows, m, sm);
        }
        for (int rr = split ? total : tid; rr < total; rr += nthr) {
            if (rr != tid) fetch(rr);
#pragma unroll
            for (int c = 0; c < NB; ++c) {
                v[c] *= sm.rinv[kb + c];  // (1 past the matrix: identity padding)
#pragma unroll
                for (int c2 = c + 1; c2 < NB; ++c2) v[c2] = fma(-v[c], sm.dg[c * DS + c2], v[c2]);
            }
#pragma unroll
            for (int c = 0; c < NB; ++c)
                if (c < bs) {
                    if (rr < rows)
                        A[(q + rr) + (int64_t)(kb + c) * n] = v[c];
                    else
                        sm.rhs[(rr - rows) * kBMaxN + kb + c] = v[c];
                }
            if (rows > 0) batch_keep_row(sm, rr < rows ? rr : rhs_row<T>(rows) + rr - rows, v);
        }
        __syncthreads();
        if (rows > 0) batch_update(sm, A, n, q, kb, rows, m);
    }
    const int fail = sm.fail;
    __syncthreads();
    return fail;
}

// L^T X = Y in place on sm.rhs for the factor in the lower triangle of A (ld = n)
// and sm.rinv: blocks from the last, one warp per right-hand side in the block,
// one thread per remaining column after it.
template <typename T>
__device__ void batch_backward(const T *A, int n, int m, BatchSmem<T> &sm) {
    constexpr int NB = kBN<T>, DS = BatchSmem<T>::kBDs;
    const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, nw = nthr >> 5;
    const int lane = tid & (NB - 1);  // (FP64: both half-warps do the same)
    for (int kb = (n - 1) / NB * NB; kb >= 0; kb -= NB) {
        const int bs = min(NB, n - kb);
        for (int e = tid; e < NB * NB; e += nthr) {
            const int r = e % NB, c = e / NB;
            if (r < bs && c < r)
                batch_fill(&sm.dg[r * DS + c], &A[(kb + r) + (int64_t)(kb + c) * n]);
            else
                sm.dg[r * DS + c] = T(0);
        }
        // the block's rows of column tid, fetched while the block is solved
        T v[NB];
        auto fetch = [&](int j) {
#pragma unroll
            for (int t = 0; t < NB; ++t) v[t] = t < bs ? A[(kb + t) + (int64_t)j * n] : T(0);
        };
        if (tid < kb) fetch(tid);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        for (int k = warp; k < m; k += nw) {
            T z = lane < bs ? sm.rhs[k * kBMaxN + kb + lane] : T(0);
            const T ri = lane < bs ? sm.rinv[kb + lane] : T(0);
#pragma unroll
            for (int c = NB - 1; c >= 0; --c) {
                const T x = shfl(z * ri, c);
                const T w = fma(-x, sm.dg[c * DS + lane], z);
                z = lane == c ? x : (lane < c ? w : z);
            }
            __syncwarp();
            if (lane < bs) sm.rhs[k * kBMaxN + kb + lane] = z;
        }
        __syncthreads();
        for (int j = tid; j < kb; j += nthr) {
            if (j != tid) fetch(j);
            for (int k = 0; k < m; ++k) {
                T s = sm.rhs[k * kBMaxN + j];
#pragma unroll
                for (int t = 0; t < NB; ++t)
                    if (t < bs) s = fma(-v[t], sm.rhs[k * kBMaxN + kb + t], s);
                sm.rhs[k * kBMaxN + j] = s;
            }
        }
        __syncthreads();
    }
}

// L L^T X = B in place for the factor in the lower triangle of A (ld = n).
template <typename T>
__device__ void batch_trsolve(const T *A, int n, T *B, int64_t ldb, int m, T *sD, T *sP) {
    const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31;
    const int nwarps = nthr >> 5;
    // ---- solve L y = b (forward), then L^T x = y (backward), 32-row blocks ----
    for (int pass = 0; pass < 2; ++pass) {
        const bool fwd = pass == 0;
        const int nblk = (n + kBNb - 1) / kBNb;
        for (int bi = 0; bi < nblk; ++bi) {
            const int kb = (fwd ? bi : nblk - 1 - bi) * kBNb;
            const int bs = min(kBNb, n - kb);
            for (int e = tid; e < 32 * 32; e += nthr) {
                const int r = e % 32, c = e / 32;
                if (r < bs && c <= r) sD[r * 33 + c] = A[(kb + r) + (int64_t)(kb + c) * n];
            }
            __syncthreads();
            // warp k solves right-hand side k on this block (lane = row)
            for (int k = warp; k < m; k += nwarps) {
                T x = (lane < bs) ? B[(kb + lane) + (int64_t)k * ldb] : T(0);
                if (fwd) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) {
                        if (c < bs) {
                            const T xc = shfl(x, c) / sD[c * 33 + c];
                            if (lane == c) x = xc;
                            if (lane > c && lane < bs) x = fma(-xc, sD[lane * 33 + c], x);
                        }
                    }
                } else {
#pragma unroll
                    for (int cc = 31; cc >= 0; --cc) {
                        if (cc < bs) {
                            const T xc = shfl(x, cc) / sD[cc * 33 + cc];
                            if (lane == cc) x = xc;
                            if (lane < cc) x = fma(-xc, sD[cc * 33 + lane], x);
                        }
                    }
                }
                if (lane < bs) B[(kb + lane) + (int64_t)k * ldb] = x;
            }
            // stage the block's coupling to the remaining rows: forward needs
            // L[r][kb+t] for r >= kb+bs, backward L[kb+t][r] for r < kb
            const int q = fwd ? kb + bs : 0, rows = fwd ? n - kb - bs : kb;
            for (int e = tid; e < rows * bs; e += nthr) {
                if (fwd) {
                    const int rr = e % rows, t = e / rows;  // consecutive rr: contiguous column
                    sP[rr * 33 + t] = A[(q + rr) + (int64_t)(kb + t) * n];
                } else {
                    const int t = e % bs, rr = e / bs;  // consecutive t: contiguous column rr
                    sP[rr * 33 + t] = A[(kb + t) + (int64_t)rr * n];
                }
            }
            __syncthreads();
            for (int e = tid; e < rows * m; e += nthr) {
                const int rr = e % rows, k = e / rows;
                T acc = B[(q + rr) + (int64_t)k * ldb];
#pragma unroll 8
                for (int t = 0; t < bs; ++t) acc = fma(-sP[rr * 33 + t], B[(kb + t) + (int64_t)k * ldb], acc);
                B[(q + rr) + (int64_t)k * ldb] = acc;
            }
            __syncthreads();
        }
    }
}

// Factor-and-solve of one system by the whole CTA: B (n x m, leading dimension
// ldb) is overwritten with X (untouched when the factorisation fails).
template <typename T>
__device__ int batch_solve_one(T *A, int n, T *B, int64_t ldb, int m, BatchSmem<T> &sm) {
    for (int e = threadIdx.x; e < n * m; e += blockDim.x) {
        const int i = e % n, k = e / n;
        batch_fill(&sm.rhs[k * kBMaxN + i], &B[i + (int64_t)k * ldb]);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    const int f = batch_factor<T>(A, n, m, sm);
    if (f >= 0) return f;
    batch_backward<T>(A, n, m, sm);
    for (int e = threadIdx.x; e < n * m; e += blockDim.x) {
        const int i = e % n, k = e / n;
        B[i + (int64_t)k * ldb] = sm.rhs[k * kBMaxN + i];
    }
    __syncthreads();
    return -1;
}

template <typename T>
__global__ void __launch_bounds__(256, 2) batch_posv_kernel(const BatchItem *__restrict__ items, int64_t count, T *Apool,
                                  T *Bpool, int32_t *info, int *counter) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BatchSmem<T> &sm = *reinterpret_cast<BatchSmem<T> *>(smem_raw);
    __shared__ int s_item;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int64_t it = s_item;
        if (it >= count) break;
        const BatchItem w = items[it];
        const int f = batch_solve_one<T>(Apool + w.a_off, w.n, Bpool + w.b_off, w.n, w.m, sm);
        if (tid == 0) info[w.idx] = f;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// f64 systems through an FP32 factorisation with FP64 refinement, per system
//
// One CTA per system, as above: the lower triangle of A (FP64, read only) is
// copied to FP32 scratch and factored there; x = 0, r = b; each iteration
// solves L L^T d = fp32(r) in FP32, adds d to x in FP64 and forms
// r = b - A x in FP64 from the lower triangle of A (one thread per row,
// sym_residual).  It stops when the normwise backward error
// max_j ||r_j|| / (||A|| ||x_j|| + ||b_j||) reaches n eps / 16, or once a
// correction no longer halves it.  A system whose FP32 factorisation breaks down, or that ends
// above 10 n eps, is solved again by the plain FP64 routine (whose verdict
// stands) from a working copy of A.  FP64 arithmetic is the scarce resource
// on this GPU: the factorisation (n^3/3) moves to the FP32 pipe and only
// 2 n^2 m per iteration stays in FP64.
constexpr int kBRefIters = 5;
// Stop at n eps / 16 (about what the plain FP64 batched solve reaches); a
// system left above 10 n eps is re-solved in plain FP64.
constexpr double kBRefTolPerN = 2.220446049250313e-16 / 16.0;
// Shared memory of the factorisations (FP32, or FP64 in the fallback) and of the
// FP32 solves ([32][33] and [kBMaxN][33] floats).
constexpr size_t kBRefSpace = (sizeof(BatchSmem<double>) + 15) / 16 * 16;
static_assert(kBRefSpace >= sizeof(BatchSmem<float>) && kBRefSpace >= 4 * (32 * 33 + kBMaxN * 33), "one space for all");
constexpr size_t kBRefScratch = (size_t)kBMaxN * kBMaxN * 8 + (size_t)kBMaxN * kBMaxRhs * (4 + 8);

// Column maxima of |X| and |R| (m <= kBMaxRhs columns each) over the CTA in one
// reduction: vx, vr hold this thread's partial maxima; on return every thread
// holds the CTA's.  red: 8 warps x 2 kBMaxRhs doubles of shared memory.
__device__ __forceinline__ void block_max_cols(double (&vx)[kBMaxRhs], double (&vr)[kBMaxRhs], double *red) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
    for (int j = 0; j < kBMaxRhs; ++j)
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            vx[j] = fmax(vx[j], __shfl_xor_sync(0xffffffffu, vx[j], o));
            vr[j] = fmax(vr[j], __shfl_xor_sync(0xffffffffu, vr[j], o));
        }
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int j = 0; j < kBMaxRhs; ++j) {
            red[warp * 2 * kBMaxRhs + j] = vx[j];
            red[warp * 2 * kBMaxRhs + kBMaxRhs + j] = vr[j];
        }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kBMaxRhs; ++j) {
        vx[j] = 0.0;
        vr[j] = 0.0;
        for (int w = 0; w < nw; ++w) {
            vx[j] = fmax(vx[j], red[w * 2 * kBMaxRhs + j]);
            vr[j] = fmax(vr[j], red[w * 2 * kBMaxRhs + kBMaxRhs + j]);
        }
    }
}

// r = B - A_sym X for the lower triangle of A (ld n), X in shared memory
// (sX[k * kBMaxRhs + j]), one thread per row: the part k <= i along row i
// (consecutive rows read consecutive addresses), the part k > i down column
// i (each thread streams its own column through L1).  M right-hand sides at
// compile time, so the scarce FP64 pipe spends no issue slot on absent
// columns and no lane waits on a shuffle reduction.
template <int M>
__device__ void sym_residual_m(const double *A, int n, const double *sX, const double *B, double *out) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double acc[M];
#pragma unroll
        for (int j = 0; j < M; ++j) acc[j] = 0.0;
        for (int k = 0; k <= i; ++k) {
            const double a = A[i + (int64_t)k * n];
#pragma unroll
            for (int j = 0; j < M; ++j) acc[j] = fma(a, sX[k * kBMaxRhs + j], acc[j]);
        }
        const double *col = A + (int64_t)i * n;
        for (int k = i + 1; k < n; ++k) {
            const double a = col[k];
#pragma unroll
            for (int j = 0; j < M; ++j) acc[j] = fma(a, sX[k * kBMaxRhs + j], acc[j]);
        }
#pragma unroll
        for (int j = 0; j < M; ++j) out[i + (int64_t)j * n] = B[i + (int64_t)j * n] - acc[j];
    }
    __syncthreads();
}

__device__ void sym_residual(const double *A, int n, const double *sX, int m, const double *B, double *out) {
    switch (m) {
        case 1: sym_residual_m<1>(A, n, sX, B, out); break;
        case 2: sym_residual_m<2>(A, n, sX, B, out); break;
        case 3: sym_residual_m<3>(A, n, sX, B, out); break;
        case 4: sym_residual_m<4>(A, n, sX, B, out); break;
        case 5: sym_residual_m<5>(A, n, sX, B, out); break;
        case 6: sym_residual_m<6>(A, n, sX, B, out); break;
        case 7: sym_residual_m<7>(A, n, sX, B, out); break;
        default: sym_residual_m<8>(A, n, sX, B, out); break;
    }
}

// out[i] = sum_k |A_sym(i, k)| (the same traversal).
__device__ void sym_rowsum(const double *A, int n, double *out) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double s = 0.0;
        for (int k = 0; k <= i; ++k) s += fabs(A[i + (int64_t)k * n]);
        const double *col = A + (int64_t)i * n;
        for (int k = i + 1; k < n; ++k) s += fabs(col[k]);
        out[i] = s;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(256, 2) batch_posv_refined_kernel(const BatchItem *__restrict__ items, int64_t count,
                                                                   const double *Apool, double *Bpool,
                                                                   int32_t *info, int *counter, char *scratch) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BatchSmem<double> &smd = *reinterpret_cast<BatchSmem<double> *>(smem_raw);  // FP64 fallback
    BatchSmem<float> &smf = *reinterpret_cast<BatchSmem<float> *>(smem_raw);    // FP32 factor (same space)
    float *sDf = (float *)smem_raw;                                             // FP32 solves (same space)
    double *sX = (double *)(smem_raw + kBRefSpace);                             // [kBMaxN][kBMaxRhs]
    __shared__ int s_item;
    __shared__ double red[8 * 2 * kBMaxRhs];
    __shared__ double s_cb[kBMaxRhs];
    const int tid = threadIdx.x, nthr = blockDim.x;
    char *base = scratch + (size_t)blockIdx.x * kBRefScratch;
    float *W = (float *)base;  // FP32 factor (ld n); the FP64 fallback's working copy uses the same space
    double *Wd = (double *)base;
    float *R32 = (float *)(base + (size_t)kBMaxN * kBMaxN * 8);
    double *R = (double *)(R32 + kBMaxN * kBMaxRhs);
    for (;;) {
        if (tid == 0) s_item = atomicAdd(counter, 1);
        __syncthreads();
        const int64_t it = s_item;
        if (it >= count) break;
        const BatchItem w = items[it];
        const int n = w.n, m = w.m;
        const double *A = Apool + w.a_off;
        double *B = Bpool + w.b_off;
        for (int64_t e = tid; e < (int64_t)n * n; e += nthr) {
            const int i = (int)(e % n), k = (int)(e / n);
            if (i >= k) W[e] = (float)A[e];
        }
        // ||A||_inf and ||b_j||_inf
        sym_rowsum(A, n, R);
        double an = 0.0;
        {
            double vb[kBMaxRhs], va[kBMaxRhs];
#pragma unroll
            for (int j = 0; j < kBMaxRhs; ++j) vb[j] = va[j] = 0.0;
            for (int i = tid; i < n; i += nthr) {
                va[0] = fmax(va[0], R[i]);
#pragma unroll
                for (int j = 0; j < kBMaxRhs; ++j)
                    if (j < m) vb[j] = fmax(vb[j], fabs(B[i + (int64_t)j * n]));
            }
            block_max_cols(vb, va, red);
            an = va[0];
#pragma unroll
            for (int j = 0; j < kBMaxRhs; ++j)
                if (tid == j) s_cb[j] = vb[j];
        }
        __syncthreads();
        const double tol = kBRefTolPerN * n;
        int f = batch_factor<float>(W, n, 0, smf);
        bool ok = f < 0;
        if (ok) {
            for (int e = tid; e < n * kBMaxRhs; e += nthr) sX[e] = 0.0;
            for (int64_t e = tid; e < (int64_t)n * m; e += nthr) R[e] = B[e];
            __syncthreads();
            double eta = INFINITY, eta_prev = INFINITY;
            for (int itr = 0; itr < kBRefIters; ++itr) {
                for (int64_t e = tid; e < (int64_t)n * m; e += nthr) R32[e] = (float)R[e];
                __syncthreads();
                batch_trsolve<float>(W, n, R32, n, m, sDf, sDf + 32 * 33);
                for (int64_t e = tid; e < (int64_t)n * m; e += nthr) {
                    const int i = (int)(e % n), j = (int)(e / n);
                    sX[i * kBMaxRhs + j] += (double)R32[e];
                }
                __syncthreads();
                sym_residual(A, n, sX, m, B, R);
                double vx[kBMaxRhs], vr[kBMaxRhs];
#pragma unroll
                for (int j = 0; j < kBMaxRhs; ++j) vx[j] = vr[j] = 0.0;
                for (int i = tid; i < n; i += nthr) {
#pragma unroll
                    for (int j = 0; j < kBMaxRhs; ++j)
                        if (j < m) {
                            vx[j] = fmax(vx[j], fabs(sX[i * kBMaxRhs + j]));
                            vr[j] = fmax(vr[j], fabs(R[i + (int64_t)j * n]));
                        }
                }
                block_max_cols(vx, vr, red);
                double e_max = 0.0;
#pragma unroll
                for (int j = 0; j < kBMaxRhs; ++j) {
                    if (j >= m) continue;
                    const double den = an * vx[j] + s_cb[j];
                    double ej = den > 0 ? vr[j] / den : (vr[j] > 0 ? INFINITY : 0.0);
                    if (ej != ej) ej = INFINITY;
                    e_max = fmax(e_max, ej);
                }
                eta = e_max;  // uniform across the CTA
                // done at the target, or once a correction no longer halves the error
                if (eta <= tol || !(eta < INFINITY) || (itr >= 1 && eta > 0.5 * eta_prev)) break;
                eta_prev = eta;
            }
            ok = eta <= 10.0 * n * 2.220446049250313e-16;
            if (ok) {
                for (int64_t e = tid; e < (int64_t)n * m; e += nthr) {
                    const int i = (int)(e % n), j = (int)(e / n);
                    B[e] = sX[i * kBMaxRhs + j];
                }
            }
        }
        if (!ok) {  // plain FP64 from a working copy of A (B still holds b)
            __syncthreads();
            for (int64_t e = tid; e < (int64_t)n * n; e += nthr) {
                const int i = (int)(e % n), k = (int)(e / n);
                if (i >= k) Wd[e] = A[e];
            }
            __syncthreads();
            f = batch_solve_one<double>(Wd, n, B, n, m, smd);
        } else {
            f = -1;
        }
        if (tid == 0) info[w.idx] = f;
        __syncthreads();
    }
}

size_t batch_refined_smem() { return kBRefSpace + sizeof(double) * kBMaxN * kBMaxRhs; }
size_t batch_refined_scratch_bytes(int ctas) { return (size_t)ctas * kBRefScratch; }

// ---------------------------------------------------------------------------
// device-resident serving loop

__device__ __forceinline__ unsigned long long ld_acquire_sys_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_sys_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Persistent CTAs of 256 threads.  Thread 0 claims the next published ticket
// (compare-and-swap on the device counter, so a ticket is claimed at most once
// and only after the host published it), the CTA copies the lower triangle of
// A into its scratch (ld = n) and solves in place with the batched routine;
// thread 0 then publishes the outcome.  Every wait is bounded: an idle CTA
// returns after idle_ns without work (the host relaunches the loop when new
// requests arrive), at once when ring->stop is set.
__global__ void __launch_bounds__(256) serve_loop_kernel(ServeRing *ring, unsigned long long *next,
                                                        double *scratch, unsigned long long idle_ns) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ long long s_ticket;
    __shared__ ServeReq s_req;
    const int tid = threadIdx.x;
    double *myA = scratch + (size_t)blockIdx.x * kBMaxN * kBMaxN;
    for (;;) {
        if (tid == 0) {
            long long claim = -1;
            const unsigned long long t_idle = globaltimer_ns();
            unsigned sleep_ns = 64;
            for (;;) {
                const unsigned long long cur = atomicAdd(next, 0ull);
                const unsigned long long pub = ld_acquire_sys_u64(&ring->published);
                if (cur < pub) {
                    if (atomicCAS(next, cur, cur + 1) == cur) {
                        claim = (long long)cur;
                        break;
                    }
                    continue;
                }
                if (*(volatile int *)&ring->stop) break;
                if (globaltimer_ns() - t_idle > idle_ns) break;
                __nanosleep(sleep_ns);
                if (sleep_ns < 2048) sleep_ns *= 2;
            }
            s_ticket = claim;
            if (claim >= 0) {
                // the host wrote the slot before it raised `published` (acquired above)
                const ServeReq *q = &ring->req[claim % kServeRing];
                s_req.A = *(void *const volatile *)&q->A;
                s_req.B = *(void *volatile *)&q->B;
                s_req.lda = *(volatile const int64_t *)&q->lda;
                s_req.ldb = *(volatile const int64_t *)&q->ldb;
                s_req.n = *(volatile const int32_t *)&q->n;
                s_req.m = *(volatile const int32_t *)&q->m;
                s_req.dtype = *(volatile const int32_t *)&q->dtype;
            }
        }
        __syncthreads();
        const long long t = s_ticket;
        if (t < 0) break;
        const ServeReq q = s_req;
        const int n = q.n;
        int f;
        if (q.dtype == 8) {
            double *W = myA;
            const double *A = (const double *)q.A;
            for (int64_t e = tid; e < (int64_t)n * n; e += blockDim.x) {
                const int i = (int)(e % n), j = (int)(e / n);
                if (i >= j) W[e] = A[i + (int64_t)j * q.lda];
            }
            __syncthreads();
            f = batch_solve_one<double>(W, n, (double *)q.B, q.ldb, q.m,
                                        *reinterpret_cast<BatchSmem<double> *>(smem_raw));
        } else {
            float *W = (float *)myA;
            const float *A = (const float *)q.A;
            for (int64_t e = tid; e < (int64_t)n * n; e += blockDim.x) {
                const int i = (int)(e % n), j = (int)(e / n);
                if (i >= j) W[e] = A[i + (int64_t)j * q.lda];
            }
            __syncthreads();
            f = batch_solve_one<float>(W, n, (float *)q.B, q.ldb, q.m,
                                       *reinterpret_cast<BatchSmem<float> *>(smem_raw));
        }
        __syncthreads();  // every thread's writes of X precede the publication
        if (tid == 0) {
            const int slot = (int)(t % kServeRing);
            __threadfence_system();
            *(volatile int32_t *)&ring->status[slot] = f >= 0 ? 1 : 0;
            *(volatile int64_t *)&ring->fail_row[slot] = f;
            st_release_sys_u64(&ring->done_seq[slot], (unsigned long long)t + 1);
        }
    }
}

size_t serve_loop_scratch_bytes(int ctas) { return (size_t)ctas * kBMaxN * kBMaxN * sizeof(double); }

int serve_loop_launch(ServeRing *ring_dev, unsigned long long *d_next, double *scratch, int ctas,
                      double idle_us, cudaStream_t st) {
    const size_t smem = sizeof(BatchSmem<double>);
    static_assert(sizeof(BatchSmem<double>) >= sizeof(BatchSmem<float>), "one space for both types");
    if (allow_dynamic_smem(serve_loop_kernel, smem) != cudaSuccess) return -1;
    LaunchScope ls(K_BATCH, st);
    serve_loop_kernel<<<(unsigned)ctas, 256, smem, st>>>(ring_dev, d_next, scratch,
                                                         (unsigned long long)(idle_us * 1e3));
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace lla

// ---------------------------------------------------------------------------
// plan, autotune cache, launch

using namespace lla;

struct lla_batch_plan {
    int64_t count = 0;
    int dtype = 8;
    std::vector<int32_t> n, m;
    std::vector<int64_t> a_off, b_off;
    int64_t a_elems = 0, b_elems = 0;
    double flops = 0.0;
    BatchItem *d_items = nullptr;
    int *d_counter = nullptr;
    int ctas_per_sm = 4, threads = 128;  // four latency chains a SM; measured best or equal at every order
    bool by_caller = false;  // the caller set the shape (kept when the mode changes, as a tuned one is not)
    bool refined = false;   // f64 systems through an FP32 factor + FP64 refinement (A read only)
    char *d_scratch = nullptr;  // per-CTA scratch of the refined mode
    std::string key;
    // graph replay cache
    cudaGraphExec_t gexec = nullptr;
    void *g_a = nullptr, *g_b = nullptr, *g_info = nullptr;
    cudaStream_t g_stream = nullptr;
};

// Generation of the batched kernels, part of the cache's keys: a shape that was measured
// with other kernels says nothing about these.  Raised with every change that moves
// their best shape.
constexpr int kBatchGeneration = 2;

static size_t batch_smem(int dtype) { return dtype == 8 ? sizeof(BatchSmem<double>) : sizeof(BatchSmem<float>); }

static bool cache_lookup(const std::string &key, int &cps, int &thr) { return lla::autotune_lookup(key, cps, thr); }
static void cache_store(const std::string &key, int cps, int thr) { lla::autotune_store(key, cps, thr); }

namespace lla {

template <typename T>
int batch_launch_raw(const BatchItem *d_items, int64_t count, T *dA, T *dB, int32_t *d_info,
                     int *d_counter, int ctas_per_sm, int threads, double flops, cudaStream_t st) {
    if (count <= 0) return 0;
    if (cudaMemsetAsync(d_counter, 0, sizeof(int), st) != cudaSuccess) return -1;
    const size_t smem = batch_smem(sizeof(T));
    if (allow_dynamic_smem(batch_posv_kernel<T>, smem) != cudaSuccess) return -1;
    const unsigned grid =
        (unsigned)std::max<int64_t>(1, std::min<int64_t>(count, (int64_t)ctas_per_sm * device_sms()));
    LaunchScope ls(K_BATCH, st, flops);
    batch_posv_kernel<T><<<grid, threads, smem, st>>>(d_items, count, dA, dB, d_info, d_counter);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template int batch_launch_raw<double>(const BatchItem *, int64_t, double *, double *, int32_t *, int *,
                                      int, int, double, cudaStream_t);
template int batch_launch_raw<float>(const BatchItem *, int64_t, float *, float *, int32_t *, int *, int,
                                     int, double, cudaStream_t);

}  // namespace lla

// The refined mode's CTAs per SM are limited by its shared memory (two fit).
static int refined_ctas_per_sm(int cps) { return std::min(cps, 2); }

template <typename T>
static cudaError_t batch_launch(lla_batch_plan *p, T *dA, T *dB, int32_t *d_info, cudaStream_t st) {
    if (p->refined && sizeof(T) == 8) {
        if (cudaMemsetAsync(p->d_counter, 0, sizeof(int), st) != cudaSuccess) return cudaGetLastError();
        const int cps = refined_ctas_per_sm(p->ctas_per_sm);
        const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(p->count, (int64_t)cps * device_sms()));
        LaunchScope ls(K_BATCH, st, p->flops);
        batch_posv_refined_kernel<<<grid, p->threads, batch_refined_smem(), st>>>(
            p->d_items, p->count, (const double *)dA, (double *)dB, d_info, p->d_counter, p->d_scratch);
        return cudaGetLastError();
    }
    if (batch_launch_raw<T>(p->d_items, p->count, dA, dB, d_info, p->d_counter, p->ctas_per_sm,
                            p->threads, p->flops, st) == 0)
        return cudaSuccess;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? cudaErrorUnknown : e;
}

extern "C" {

int lla_batch_plan_create(int64_t count, const int32_t *n, const int32_t *m, int elem_bytes,
                          lla_batch_plan **out, lla_error *err) {
    if (!out || count < 0 || (count > 0 && (!n || !m)) || (elem_bytes != 4 && elem_bytes != 8))
        return lla__set_status(err, LLA_ERR_INVALID_ARG);
    for (int64_t i = 0; i < count; ++i) {
        if (n[i] < 0 || m[i] < 0) return lla__set_status(err, LLA_ERR_INVALID_ARG);
        if (n[i] > kBMaxN || m[i] > kBMaxRhs) return lla__set_status(err, LLA_ERR_TOO_LARGE);
    }
    lla__set_status(err, LLA_OK);
    lla_batch_plan *p = new lla_batch_plan();
    p->count = count;
    p->dtype = elem_bytes;
    p->n.assign(n, n + count);
    p->m.assign(m, m + count);
    p->a_off.resize(count);
    p->b_off.resize(count);
    // pools in submission order, each system 16-byte aligned
    const int64_t align = 16 / elem_bytes;
    int64_t ao = 0, bo = 0;
    int hist[9] = {0};
    int maxm = 0;
    for (int64_t i = 0; i < count; ++i) {
        p->a_off[i] = ao;
        p->b_off[i] = bo;
        ao += ((int64_t)n[i] * n[i] + align - 1) / align * align;
        bo += ((int64_t)n[i] * m[i] + align - 1) / align * align;
        p->flops += (double)n[i] * n[i] * n[i] / 3.0 + 2.0 * n[i] * n[i] * m[i];
        int b = 0;
        while ((32 << b) < n[i] && b < 8) ++b;
        hist[b]++;
        maxm = std::max(maxm, (int)m[i]);
    }
    p->a_elems = ao;
    p->b_elems = bo;
    // work list: largest systems first
    std::vector<BatchItem> items(count);
    for (int64_t i = 0; i < count; ++i)
        items[i] = BatchItem{n[i], m[i], (int32_t)i, 0, p->a_off[i], p->b_off[i]};
    std::stable_sort(items.begin(), items.end(), [](const BatchItem &a, const BatchItem &b) {
        const double ca = (double)a.n * a.n * (a.n + 6.0 * a.m), cb = (double)b.n * b.n * (b.n + 6.0 * b.m);
        return ca > cb;
    });
    // autotune-cache key: the kernels' generation, element size, count, size-bucket histogram,
    // widest RHS
    char key[256];
    std::snprintf(key, sizeof(key), "k%d:b%d:c%lld:h%d-%d-%d-%d-%d-%d-%d-%d-%d:m%d",
                  kBatchGeneration, elem_bytes, (long long)count, hist[0], hist[1], hist[2], hist[3], hist[4], hist[5], hist[6],
                  hist[7], hist[8], maxm);
    p->key = key;
    int cps, thr;
    if (cache_lookup(p->key, cps, thr)) {
        p->ctas_per_sm = cps;
        p->threads = thr;
    }
    cudaError_t e = cudaMalloc(&p->d_items, sizeof(BatchItem) * std::max<int64_t>(1, count));
    if (e == cudaSuccess) e = cudaMalloc(&p->d_counter, sizeof(int));
    if (e == cudaSuccess && count > 0)
        e = cudaMemcpy(p->d_items, items.data(), sizeof(BatchItem) * count, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        const size_t smem = batch_smem(elem_bytes);
        e = elem_bytes == 8 ? allow_dynamic_smem(batch_posv_kernel<double>, smem)
                            : allow_dynamic_smem(batch_posv_kernel<float>, smem);
    }
    if (e != cudaSuccess) {
        cudaFree(p->d_items);
        cudaFree(p->d_counter);
        delete p;
        return lla__set_cuda_error(err, e);
    }
    *out = p;
    return LLA_OK;
}

void lla_batch_plan_destroy(lla_batch_plan *p) {
    if (!p) return;
    if (p->gexec) cudaGraphExecDestroy(p->gexec);
    if (p->d_scratch) cudaFree(p->d_scratch);
    cudaFree(p->d_items);
    cudaFree(p->d_counter);
    delete p;
}

int lla_batch_plan_info(const lla_batch_plan *p, int64_t *a_elems, int64_t *b_elems, int64_t *a_off,
                        int64_t *b_off, int *ctas_per_sm, int *threads, double *flops) {
    if (!p) return LLA_ERR_INVALID_ARG;
    if (a_elems) *a_elems = p->a_elems;
    if (b_elems) *b_elems = p->b_elems;
    if (a_off) std::memcpy(a_off, p->a_off.data(), sizeof(int64_t) * p->count);
    if (b_off) std::memcpy(b_off, p->b_off.data(), sizeof(int64_t) * p->count);
    if (ctas_per_sm) *ctas_per_sm = p->ctas_per_sm;
    if (threads) *threads = p->threads;
    if (flops) *flops = p->flops;
    return LLA_OK;
}

static void apply_shape(lla_batch_plan *p, int ctas_per_sm, int threads) {
    if (p->ctas_per_sm == ctas_per_sm && p->threads == threads) return;
    p->ctas_per_sm = ctas_per_sm;
    p->threads = threads;
    if (p->gexec) {
        cudaGraphExecDestroy(p->gexec);
        p->gexec = nullptr;
    }
}

int lla_batch_set_shape(lla_batch_plan *p, int ctas_per_sm, int threads) {
    if (!p || ctas_per_sm < 1 || ctas_per_sm > 8 || (threads != 128 && threads != 256))
        return LLA_ERR_INVALID_ARG;
    p->by_caller = true;
    apply_shape(p, ctas_per_sm, threads);
    return LLA_OK;
}

// Switches an f64 plan between the plain FP64 solve (A factored in place) and
// the FP32 factorisation with per-system FP64 refinement (A read only).
int lla_batch_set_refined(lla_batch_plan *p, int refined, lla_error *err) {
    if (!p || (refined && p->dtype != 8)) return lla__set_status(err, LLA_ERR_INVALID_ARG);
    lla__set_status(err, LLA_OK);
    const bool want = refined != 0;
    if (want && !p->d_scratch) {
        cudaError_t e = allow_dynamic_smem(batch_posv_refined_kernel, batch_refined_smem());
        if (e == cudaSuccess) e = cudaMalloc(&p->d_scratch, batch_refined_scratch_bytes(2 * device_sms()));
        if (e != cudaSuccess) {
            p->d_scratch = nullptr;
            return lla__set_cuda_error(err, e);
        }
    }
    if (p->refined != want) {
        p->refined = want;
        if (p->gexec) {
            cudaGraphExecDestroy(p->gexec);
            p->gexec = nullptr;
        }
        // the launch shape is cached per mode
        p->key += want ? ":r" : "";
        if (!want && p->key.size() > 2 && p->key.compare(p->key.size() - 2, 2, ":r") == 0)
            p->key.resize(p->key.size() - 2);
        int cps, thr;
        if (cache_lookup(p->key, cps, thr)) {
            p->ctas_per_sm = cps;
            p->threads = thr;
        } else if (!p->by_caller) {  // two CTAs of the refined kernel fit an SM
            p->ctas_per_sm = want ? 2 : 4;
            p->threads = want ? 256 : 128;
        }
    }
    return LLA_OK;
}

static int batch_posv(lla_batch_plan *p, void *dA, void *dB, int32_t *d_info, void *stream,
                      lla_error *err, int elem_bytes) {
    if (!p || p->dtype != elem_bytes || (p->count > 0 && (!dA || !dB || !d_info)))
        return lla__set_status(err, LLA_ERR_INVALID_ARG);
    lla__set_status(err, LLA_OK);
    if (p->count == 0) return LLA_OK;
    cudaError_t e = elem_bytes == 8
                        ? batch_launch<double>(p, (double *)dA, (double *)dB, d_info, (cudaStream_t)stream)
                        : batch_launch<float>(p, (float *)dA, (float *)dB, d_info, (cudaStream_t)stream);
    return e == cudaSuccess ? LLA_OK : lla__set_cuda_error(err, e);
}

int lla_dbatch_posv_device(lla_batch_plan *p, double *dA, double *dB, int32_t *d_info, void *stream,
                           lla_error *err) {
    return batch_posv(p, dA, dB, d_info, stream, err, 8);
}

int lla_sbatch_posv_device(lla_batch_plan *p, float *dA, float *dB, int32_t *d_info, void *stream,
                           lla_error *err) {
    return batch_posv(p, dA, dB, d_info, stream, err, 4);
}

// Same work as lla_?batch_posv_device, replayed from a CUDA graph: the first
// call for a given (pools, info, stream) captures [counter reset, persistent
// kernel] and instantiates it; later calls launch the executable graph.
int lla_batch_posv_graph(lla_batch_plan *p, void *dA, void *dB, int32_t *d_info, void *stream,
                         lla_error *err) {
    if (!p || (p->count > 0 && (!dA || !dB || !d_info))) return lla__set_status(err, LLA_ERR_INVALID_ARG);
    lla__set_status(err, LLA_OK);
    if (p->count == 0) return LLA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e;
    if (!p->gexec || p->g_a != dA || p->g_b != dB || p->g_info != d_info || p->g_stream != st) {
        if (p->gexec) {
            cudaGraphExecDestroy(p->gexec);
            p->gexec = nullptr;
        }
        cudaStream_t cap = nullptr;
        if ((e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking)) != cudaSuccess)
            return lla__set_cuda_error(err, e);
        cudaGraph_t g = nullptr;
        e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            prof_capturing() = true;
            const cudaError_t le = p->dtype == 8
                                       ? batch_launch<double>(p, (double *)dA, (double *)dB, d_info, cap)
                                       : batch_launch<float>(p, (float *)dA, (float *)dB, d_info, cap);
            prof_capturing() = false;
            e = cudaStreamEndCapture(cap, &g);
            if (le != cudaSuccess) e = le;
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&p->gexec, g, 0);
        if (g) cudaGraphDestroy(g);
        cudaStreamDestroy(cap);
        if (e != cudaSuccess) return lla__set_cuda_error(err, e);
        p->g_a = dA;
        p->g_b = dB;
        p->g_info = d_info;
        p->g_stream = st;
    }
    {
        // one kernel per replay (plus the counter reset): counted and timed like a launch
        LaunchScope ls(K_BATCH, st, p->flops);
        e = cudaGraphLaunch(p->gexec, st);
    }
    return e == cudaSuccess ? LLA_OK : lla__set_cuda_error(err, e);
}

// Times every (CTAs per SM, threads) candidate on the caller's batch (A and B
// are restored from copies between trials, so the pools keep their inputs),
// keeps the fastest and appends it to the autotune cache file
// (LLA_AUTOTUNE_CACHE, default ~/.cache/lla_gb300_autotune.txt) under the
// batch's shape key.  best_ms (optional) receives the winner's time.
int lla_batch_autotune(lla_batch_plan *p, void *dA, void *dB, int32_t *d_info, void *stream,
                       double *best_ms, lla_error *err) {
    if (!p || (p->count > 0 && (!dA || !dB || !d_info))) return lla__set_status(err, LLA_ERR_INVALID_ARG);
    lla__set_status(err, LLA_OK);
    if (p->count == 0) return LLA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t abytes = (size_t)p->a_elems * p->dtype, bbytes = (size_t)p->b_elems * p->dtype;
    void *a0 = nullptr, *b0 = nullptr;
    cudaError_t e = cudaMalloc(&a0, abytes);
    if (e == cudaSuccess) e = cudaMalloc(&b0, bbytes);
    if (e == cudaSuccess) e = cudaMemcpyAsync(a0, dA, abytes, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(b0, dB, bbytes, cudaMemcpyDeviceToDevice, st);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    const int cands[][2] = {{1, 256}, {2, 256}, {3, 256}, {2, 128}, {3, 128}, {4, 128}};
    int best_c = p->ctas_per_sm, best_t = p->threads;
    float best = 1e30f;
    const size_t smem = batch_smem(p->dtype);
    for (const auto &c : cands) {
        if (e != cudaSuccess) break;
        if (smem * c[0] > 227 * 1024) continue;  // does not fit on one SM
        if (p->refined && c[0] > 2) continue;      // the refined kernel fits two CTAs per SM
        p->ctas_per_sm = c[0];
        p->threads = c[1];
        float tbest = 1e30f;
        for (int rep = 0; rep < 2 && e == cudaSuccess; ++rep) {
            e = cudaMemcpyAsync(dA, a0, abytes, cudaMemcpyDeviceToDevice, st);
            if (e == cudaSuccess) e = cudaMemcpyAsync(dB, b0, bbytes, cudaMemcpyDeviceToDevice, st);
            if (e == cudaSuccess) e = cudaEventRecord(e0, st);
            if (e == cudaSuccess)
                e = p->dtype == 8 ? batch_launch<double>(p, (double *)dA, (double *)dB, d_info, st)
                                  : batch_launch<float>(p, (float *)dA, (float *)dB, d_info, st);
            if (e == cudaSuccess) e = cudaEventRecord(e1, st);
            if (e == cudaSuccess) e = cudaEventSynchronize(e1);
            float ms = 0.f;
            if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
            if (e == cudaSuccess) tbest = std::min(tbest, ms);
        }
        if (e == cudaSuccess && tbest < best) {
            best = tbest;
            best_c = c[0];
            best_t = c[1];
        }
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(dA, a0, abytes, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dB, b0, bbytes, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(a0);
    cudaFree(b0);
    apply_shape(p, best_c, best_t);
    if (e != cudaSuccess) return lla__set_cuda_error(err, e);
    cache_store(p->key, best_c, best_t);
    if (best_ms) *best_ms = best;
    return LLA_OK;
}

}  // extern "C"
