// lla_potrf.cu -- blocked Cholesky factorisation kernels (lower triangle,
// column-major device matrices), EXACT mode.  It keeps the reference's
// per-element operation order (src/cholesky.rs:54-74): for every pair j > k the sum
//     s_jk = sum_{i<k} L[k,i] * L[j,i]
// is accumulated from zero in ascending i, then
//     L[j,k] = (A[j,k] - s_jk) / L[k,k],      d_j += L[j,k]^2   (ascending k),
//     L[j,j] = sqrt(A[j,j] - d_j)             (error when the pivot is <= 0).
// The reference evaluates these row by row; here the same sums are grown
// right-looking, one panel of columns at a time, in separate accumulator
// arrays S (n x n, lower part used) and D (n).  Every accumulator receives
// exactly the same products in exactly the same order, each multiply and add
// rounded separately, so the factor is bit-identical to the reference's.
//
// FAST mode is in lla_fast_chol.cu.
#include "lla_common.cuh"
#include "lla_int_math.h"
#include "lla_kernels.h"
#include "lla_prof.h"

namespace lla {

// ---------------------------------------------------------------------------
// EXACT kernels.  An FP64 instruction takes 64 cycles of its sub-partition
// whatever its active lanes, and a library root or division about nine of them,
// so: roots and quotients run in integer arithmetic (lla_int_math.h,
// bit-identical to IEEE), the accumulators stay in registers as patches of 16
// rows x 2 columns, and tiles are small, so that every SM's pipe has a share.
// Per panel of a 512 x 512 factorisation: diagonal block 18 us, panel 15, update 10
// (f64; the whole factor 730 us).  With the library's roots and divisions, sums in
// shared memory and 64 x 64 tiles: 53, 66, 82 (3160 us).
constexpr int kNbExact = 32;

// Asynchronous copy to shared memory: all of a thread's copies are in flight at once.
template <typename T>
__device__ __forceinline__ void exact_copy(T *dst, const T *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(sizeof(T))
                 : "memory");
}

// d <= 0 as the reference tests it (src/cholesky.rs:69, false for NaN).
template <typename T>
__device__ __forceinline__ bool exact_not_positive(T d) {
    return d <= T(0);
}

// Root and quotients of the reference (src/cholesky.rs:62, 73) for one pivot.
// LIB: the library's functions, for whatever the integer ones do not take (a
// pivot that is not a positive normal number, quotients outside the comfortable
// exponent range); a kernel runs the integer form first, without a branch on its
// chain, and the other only if some ok came back false.
template <typename T, bool LIB>
struct ExactPivot {
    T l;
    __device__ __forceinline__ void from_square(T dd, bool &ok) { l = Arith<T>::sqrt_(dd); }
    __device__ __forceinline__ void from_root(T v) { l = v; }
    __device__ __forceinline__ T divide(T t, bool &ok) const { return Arith<T>::div(t, l); }
};
template <>
struct ExactPivot<double, false> {
    double l;
    ImDivisor q;
    __device__ __forceinline__ void from_square(double dd, bool &ok) {
        ok = ok && im_positive_normal(im_bits(dd));
        l = im_sqrt(dd, q);
    }
    __device__ __forceinline__ void from_root(double v) {
        l = v;
        q = im_divisor(v);
    }
    __device__ __forceinline__ double divide(double t, bool &ok) const {
        bool good;
        const double x = im_div(t, q, good);
        ok = ok && good;
        return x;
    }
};

// Diagonal block [p, p+b), b <= 32, one CTA.  Warp 0 (lane = row) walks the
// chain, one column ahead of the others: it adds column k's products to the sums
// of column k + 1, takes the pivot and divides; it also keeps the diagonal sums
// D.  The warps of the other sub-partitions hold the sums of the columns right of
// it in registers and hand column k + 2 over once column k is in it.  One barrier
// per column.
constexpr int kExDiagThreads = 512;
constexpr int kExPatches = 24, kExPatchWarps = 12, kExSlots = 2;

// Returns (to every thread) whether the block stands; with LIB always, and
// *s_fail is the failing column or -1.
template <typename T, bool LIB>
__device__ bool exact_diag_block(const T *W, const T *S, const T *D, int64_t ld, int64_t p, int b,
                                 T (*a)[kNbExact + 1], T (*s)[kNbExact + 1], int64_t failed, int *s_fail) {
    using Ar = Arith<T>;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    for (int e = tid; e < kNbExact * kNbExact; e += kExDiagThreads) {
        const int r = e % kNbExact, c = e / kNbExact;
        // a short block is padded with the identity
        if (r < b && c <= r)
            exact_copy(&a[c][r], &cm(W, ld, p + r, p + c));
        else
            a[c][r] = T(r == c ? 1 : 0);
        if (r < b && c < r && p > 0)
            exact_copy(&s[c][r], &cm(S, ld, p + r, p + c));
        else
            s[c][r] = T(0);
    }
    if (tid == 0) *s_fail = -1;
    T d = (warp == 0 && lane < b && p > 0) ? D[p + lane] : T(0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (failed >= 0) return true;  // (the same for all threads; tested here, its load in flight with the others)
    __syncthreads();
    const bool upd = (warp & 3) != 0;
    T acc[kExSlots];
    int row[kExSlots], col[kExSlots];  // col < 0: no patch
    if (upd) {
#pragma unroll
        for (int i = 0; i < kExSlots; ++i) {
            // rightmost columns first: pairs 15 .. 8 of rows 16-31, then pairs 7 .. 0 of both row groups
            const int t = warp - 1 - (warp >> 2) + kExPatchWarps * i;
            const int j = t < 8 ? 15 - t : 7 - (t - 8) / 2, g = t < 8 ? 1 : 1 - (t & 1);
            row[i] = 16 * g + (lane & 15);
            col[i] = t < kExPatches ? 2 * j + (lane >> 4) : -1;
            acc[i] = t < kExPatches ? s[col[i]][row[i]] : T(0);
        }
    }
    bool bad = false, ok = true;
    T lk = T(0);  // warp 0: this row's entry of the last finished column
    // warp 0: column c, whose sums hold all products of columns before c - 1
    auto finish = [&](int c) {
        T sum = s[c][lane];
        const T av = a[c][lane], ac = a[c][c];
        d = Ar::add(d, Ar::mul(lk, lk));                           // (:64) for column c - 1 (0 before the first)
        const T dd = Ar::sub(ac, __shfl_sync(0xffffffffu, d, c));  // d = A[j,j] - d  (:66)
        if (c > 0) {
            const T lc = __shfl_sync(0xffffffffu, lk, c);  // L[c, c-1]
            sum = Ar::add(sum, Ar::mul(lc, lk));           // (:59-61), term c - 1
        }
        const T t = Ar::sub(av, sum);
        if (LIB && exact_not_positive(dd)) {  // (:69)
            bad = true;
            if (lane == 0) *s_fail = c;
            return;
        }
        ExactPivot<T, LIB> piv;
        bool good = true;
        piv.from_square(dd, ok);  // (:73)
        const T l = piv.divide(t, good);  // (:62)
        ok = ok && (good || lane <= c);
        lk = lane > c ? l : T(0);
        if (lane >= c) a[c][lane] = lane == c ? piv.l : l;
    };
    if (warp == 0) finish(0);
    for (int k = 0;; ++k) {
        __syncthreads();  // column k is final
        // a failure at column k ends the loop here for everyone; one at column k + 1, which warp 0
        // may already have recorded, after the next barrier
        if (LIB && warp > 0) bad = (unsigned)*(volatile int *)s_fail <= (unsigned)k;
        if (bad || k == kNbExact - 1) break;
        if (warp == 0) {
            finish(k + 1);
        } else if (upd) {
#pragma unroll
            for (int i = 0; i < kExSlots; ++i) {
                if ((col[i] | 1) < k + 2) break;  // (the same for the whole warp)
                const T u = Ar::add(acc[i], Ar::mul(a[k][col[i]], a[k][row[i]]));
                if (col[i] >= k + 2) acc[i] = u;
                if (col[i] == k + 2) s[k + 2][row[i]] = u;
            }
        }
    }
    return __syncthreads_and(ok) != 0;
}

template <typename T>
__global__ void __launch_bounds__(kExDiagThreads) potrf_exact_diag(T *W, const T *S, const T *D, int64_t ld,
                                                                 int64_t p, int b, int64_t *info) {
    __shared__ T a[kNbExact][kNbExact + 1];  // [column][row]: A, then L
    __shared__ T s[kNbExact][kNbExact + 1];  // sums
    __shared__ int s_fail;
    const int tid = threadIdx.x;
    pdl_wait();
    pdl_trigger();
    const int64_t failed = *(volatile int64_t *)info;  // an earlier panel failed
    constexpr bool lib = sizeof(T) == 4;  // FP32 roots and quotients are fast as they are
    if (!exact_diag_block<T, lib>(W, S, D, ld, p, b, a, s, failed, &s_fail) && !lib)
        exact_diag_block<T, true>(W, S, D, ld, p, b, a, s, failed, &s_fail);
    if (failed >= 0) return;
    if (s_fail >= 0 && tid == 0) *info = p + s_fail;
    // every value computed (on failure the caller keeps only rows < info and row
    // info's strict lower part)
    for (int e = tid; e < kNbExact * kNbExact; e += kExDiagThreads) {
        const int r = e % kNbExact, c = e / kNbExact;
        if (r < b && c <= r) cm(W, ld, p + r, p + c) = a[c][r];
    }
}

// Rows [q, n) below the diagonal block, q = p + 32; 16 rows per CTA.  The sums
// stay in registers as patches of 8 rows x 4 columns, two per warp (warp w: rows
// 8 (w % 2) .., column quads w / 2 and w / 2 + 4); quads are finished in turn by
// their two owners, one barrier each, the next owners bringing their own quad up to
// date first.  The chain of divisions and sums bounds it: 15 us a panel; 17 by pairs of
// columns, with twice the barriers (one copy of the division in a rolled loop: 16, and
// the diagonal block so 20 instead of 18).  Warp 8 adds the rows' squares to D as their columns appear.
constexpr int kExRows = 16;
constexpr int kExPanelThreads = 288;

template <typename T, bool LIB>
__device__ bool exact_panel_rows(const T *W, const T *S, const T *D, int64_t ld, int64_t n, int64_t p, int64_t j0,
                                 const T (*l11)[kNbExact + 1], const ExactPivot<T, LIB> *piv, T (*x)[kExRows], T &dj) {
    using Ar = Arith<T>;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c4 = lane >> 3, wq = warp >> 1;
    const int row = warp < 8 ? 8 * (warp & 1) + (lane & 7) : lane & 15;
    const bool in = j0 + row < n;
    T av[2] = {T(0), T(0)}, sv[2] = {T(0), T(0)};
    if (warp < 8) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int64_t c = p + 4 * (wq + 4 * i) + c4;
            av[i] = in ? cm(W, ld, j0 + row, c) : T(0);
            sv[i] = (in && p > 0) ? cm(S, ld, j0 + row, c) : T(0);
        }
    }
    dj = (warp == 8 && in && p > 0) ? D[j0 + row] : T(0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();  // l11, piv
    bool ok = true;
    auto solve = [&](int q, T a0, T s0) {  // column quad q
        const int c = 4 * q;
        const ExactPivot<T, LIB> pv = piv[c + c4];
        const T l0 = l11[c][c + c4], l1 = l11[c + 1][c + c4], l2 = l11[c + 2][c + c4];
        // (a lane's sum goes on past its own column; nothing reads it there)
        bool g[4] = {true, true, true, true};
        const T u0 = pv.divide(Ar::sub(a0, s0), g[0]);  // (:62)
        s0 = Ar::add(s0, Ar::mul(l0, __shfl_sync(0xffffffffu, u0, lane & 7)));
        const T u1 = pv.divide(Ar::sub(a0, s0), g[1]);
        s0 = Ar::add(s0, Ar::mul(l1, __shfl_sync(0xffffffffu, u1, 8 + (lane & 7))));
        const T u2 = pv.divide(Ar::sub(a0, s0), g[2]);
        s0 = Ar::add(s0, Ar::mul(l2, __shfl_sync(0xffffffffu, u2, 16 + (lane & 7))));
        const T u3 = pv.divide(Ar::sub(a0, s0), g[3]);
        x[c + c4][row] = c4 & 2 ? (c4 & 1 ? u3 : u2) : (c4 & 1 ? u1 : u0);
        ok = ok && (c4 & 2 ? (c4 & 1 ? g[3] : g[2]) : (c4 & 1 ? g[1] : g[0]));
    };
    if (wq == 0) solve(0, av[0], sv[0]);
    __syncthreads();
#pragma unroll
    for (int i0 = 0; i0 < 2; ++i0) {
#pragma unroll 1
        for (int w0 = 0; w0 < 4; ++w0) {
            const int j = 4 * i0 + w0;  // quad j is finished: add its products to the quads right of it
            T xv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) xv[u] = x[4 * j + u][row];
            if (warp == 8) {
#pragma unroll
                for (int u = 0; u < 4; ++u) dj = Ar::add(dj, Ar::mul(xv[u], xv[u]));  // (:64)
            } else {
#pragma unroll
                for (int i = i0; i < 2; ++i) {
                    const int q = 4 * i + wq;
                    if (q <= j) continue;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        sv[i] = Ar::add(sv[i], Ar::mul(l11[4 * j + u][4 * q + c4], xv[u]));  // (:59-61)
                    if (q == j + 1) solve(q, av[i], sv[i]);
                }
            }
            if (j < kNbExact / 4 - 1) __syncthreads();
        }
    }
    return __syncthreads_and(ok) != 0;
}

template <typename T>
__global__ void __launch_bounds__(kExPanelThreads) potrf_exact_panel(T *W, const T *S, T *D, int64_t ld, int64_t n,
                                                                   int64_t p, const int64_t *info) {
    constexpr bool lib = sizeof(T) == 4;
    __shared__ T l11[kNbExact][kNbExact + 1];  // [column][row]
    __shared__ T x[kNbExact][kExRows];         // finished columns
    __shared__ ExactPivot<T, lib> piv[kNbExact];
    __shared__ ExactPivot<T, true> lpiv[kNbExact];
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t j0 = p + kNbExact + (int64_t)blockIdx.x * kExRows;
    pdl_wait();
    pdl_trigger();
    const int64_t failed = *(volatile const int64_t *)info;  // (its load in flight with the others)
#pragma unroll
    for (int e = tid; e < kNbExact * kNbExact; e += kExPanelThreads) {
        const int r = e % kNbExact, c = e / kNbExact;
        if (c <= r) exact_copy(&l11[c][r], &cm(W, ld, p + r, p + c));
    }
    if (tid < kNbExact) {
        const T l = cm(W, ld, p + tid, p + tid);
        piv[tid].from_root(l);
        lpiv[tid].from_root(l);
    }
    if (failed >= 0) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    T dj;
    if (!exact_panel_rows<T, lib>(W, S, D, ld, n, p, j0, l11, piv, x, dj) && !lib)
        exact_panel_rows<T, true>(W, S, D, ld, n, p, j0, l11, lpiv, x, dj);
    for (int e = tid; e < kExRows * kNbExact; e += kExPanelThreads) {
        const int r = e % kExRows, c = e / kExRows;
        if (j0 + r < n) cm(W, ld, j0 + r, p + c) = x[c][r];
    }
    if (tid >> 5 == 8 && lane < kExRows && j0 + lane < n) D[j0 + lane] = dj;
}

// Lower-triangular tile enumeration: t -> (I, J) with J <= I.
__device__ __forceinline__ void tri_tile(int64_t t, int64_t &I, int64_t &J) {
    int64_t i = (int64_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((i + 1) * (i + 2) / 2 <= t) ++i;
    while (i * (i + 1) / 2 > t) --i;
    I = i;
    J = t - i * (i + 1) / 2;
}

// S[j, k2] += L[k2, k] L[j, k] for the panel's 32 columns in ascending k, each
// product and sum rounded separately, on 16 x 16 tiles of the strictly lower
// part of [q, n)^2 (the FP64 pipe of one SM needs 64 us for a 64 x 64 tile, so
// small tiles spread it).  Thread (row r16, columns 4 w + cc, + 2) of warp w.
constexpr int kExTile = 16;

template <typename T>
__global__ void __launch_bounds__(128) potrf_exact_update(const T *W, T *S, int64_t ld, int64_t n, int64_t p,
                                                         const int64_t *info) {
    using Ar = Arith<T>;
    __shared__ T lj[kNbExact][kExTile];  // [k][row]
    __shared__ T lk[kNbExact][kExTile];
    pdl_wait();
    pdl_trigger();
    const int64_t failed = *(volatile const int64_t *)info;  // (its load in flight with the others)
    int64_t I, J;
    tri_tile(blockIdx.x, I, J);
    const int64_t q = p + kNbExact, j0 = q + I * kExTile, k0 = q + J * kExTile;
    const int tid = threadIdx.x, lane = tid & 31, r16 = lane & 15, c0 = 4 * (tid >> 5) + (lane >> 4);
    T acc[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int64_t j = j0 + r16, k2 = k0 + c0 + 2 * i;
        acc[i] = (j < n && k2 < j && p > 0) ? cm(S, ld, j, k2) : T(0);
    }
#pragma unroll
    for (int e = tid; e < kExTile * kNbExact; e += 128) {
        const int r = e % kExTile, k = e / kExTile;
        lj[k][r] = (j0 + r < n) ? cm(W, ld, j0 + r, p + k) : T(0);
        lk[k][r] = (k0 + r < n) ? cm(W, ld, k0 + r, p + k) : T(0);
    }
    if (failed >= 0) return;
    __syncthreads();
#pragma unroll 8
    for (int k = 0; k < kNbExact; ++k)
#pragma unroll
        for (int i = 0; i < 2; ++i) acc[i] = Ar::add(acc[i], Ar::mul(lk[k][c0 + 2 * i], lj[k][r16]));
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int64_t j = j0 + r16, k2 = k0 + c0 + 2 * i;
        if (j < n && k2 < j) cm(S, ld, j, k2) = acc[i];
    }
}

// ---------------------------------------------------------------------------
// Host drivers.

static int64_t tri_tiles(int64_t m, int tile) {
    const int64_t t = ceil_div(m, tile);
    return t * (t + 1) / 2;
}

template <typename T>
int potrf_exact_launch(T *W, T *S, T *D, int64_t n, int64_t ld, int64_t *d_info,
                       cudaStream_t st) {
    // The sums S (n x n, ld) and D (n) start at zero: the first panel's kernels
    // (p == 0) take them as zero and write them, so they need no clearing.
    for (int64_t p = 0; p < n; p += kNbExact) {
        const int b = (int)std::min<int64_t>(kNbExact, n - p);
        {
            LaunchScope ls(K_POTRF_EXACT_DIAG, st, (double)b * b * b / 3.0);
            launch_maybe_pdl(p > 0, potrf_exact_diag<T>, dim3(1), dim3(kExDiagThreads), 0, st, W, (const T *)S,
                             (const T *)D, ld, p, b, d_info);
        }
        const int64_t rest = n - p - b;
        if (rest > 0) {
            {
                LaunchScope ls(K_POTRF_EXACT_PANEL, st, (double)rest * b * b);
                launch_maybe_pdl(true, potrf_exact_panel<T>, dim3((unsigned)ceil_div(rest, kExRows)),
                                 dim3(kExPanelThreads), 0, st, W, (const T *)S, D, ld, n, p, (const int64_t *)d_info);
            }
            LaunchScope ls(K_POTRF_EXACT_UPDATE, st, (double)rest * (rest - 1) * b);
            launch_maybe_pdl(true, potrf_exact_update<T>, dim3((unsigned)tri_tiles(rest, kExTile)), dim3(128), 0, st,
                             (const T *)W, S, ld, n, p, (const int64_t *)d_info);
        }
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template int potrf_exact_launch<double>(double *, double *, double *, int64_t, int64_t, int64_t *,
                                        cudaStream_t);
template int potrf_exact_launch<float>(float *, float *, float *, int64_t, int64_t, int64_t *,
                                       cudaStream_t);
}  // namespace lla
