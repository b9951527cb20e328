// lla_lobpcg.cu -- tall-skinny products of LOBPCG's Cholesky-QR
// (src/lobpcg/algorithm.rs:63-96): the Gram matrices V^T V and Y^T V, and the
// constraint update V -= Y U.  The Cholesky of the small Gram matrix and the
// triangular solve with it reuse the library's factor and substitution kernels
// (lla_api.cpp).
//
// C = A^T B for tall A (n x ka) and B (n x kb), column-major: the rows are cut
// into fixed chunks; a CTA sums its chunk's products in FP64/FP32 FMA, and a
// second kernel adds the chunk partials in a fixed order, so the result is
// deterministic (independent of scheduling).  Up to 2048 outputs (of a symmetric
// product only the lower ones count) are dealt out one by one to the CTA's
// threads, so that no lane of the scarce FP64 pipe works on padding, and about
// two chunks per SM share the rows; larger products go in 32 x 32 tiles, a CTA
// each.  V^T V of 40000 x 20: 313 us in tiles (40 CTAs, 1024 outputs where 210
// count) -> 32 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "lla_common.cuh"
#include "lla_int_math.h"
#include "lla_kernels.h"
#include "lla_prof.h"

namespace lla {

constexpr int kAtbTile = 32;
constexpr int64_t kAtbRows = 1024;  // rows per chunk
constexpr int kAtbMaxChunks = 64;

// Outputs of a product, and whether they are dealt out one by one.
constexpr int64_t kAtbPacked = 2048;
constexpr int64_t kAtbPackedRows = 32;      // rows staged at a time
constexpr int64_t kAtbPackedChunks = 304;   // about two CTAs per SM
static int64_t atb_outputs(int64_t ka, int64_t kb, int symmetric) { return symmetric ? ka * (ka + 1) / 2 : ka * kb; }
static bool atb_packed(int64_t ka, int64_t kb, int symmetric) {
    // the staged rows of both operands fit shared memory in FP64: (ka + kb) * 32 * 8 bytes
    return atb_outputs(ka, kb, symmetric) <= kAtbPacked && ka + kb <= 160;
}

static int64_t atb_chunks(int64_t n, int64_t ka, int64_t kb, int symmetric) {
    const bool packed = atb_packed(ka, kb, symmetric);
    const int64_t rows = packed ? 4 * kAtbPackedRows : kAtbRows, most = packed ? kAtbPackedChunks : kAtbMaxChunks;
    return std::min(most, std::max<int64_t>(1, (n + rows - 1) / rows));
}

size_t atb_ws_elems(int64_t n, int64_t ka, int64_t kb) {
    return (size_t)std::max(atb_chunks(n, ka, kb, 0), atb_chunks(n, ka, kb, ka == kb ? 1 : 0)) * ka * kb;
}

// Partial P[z] = A[rows of chunk z]^T B[rows of chunk z], output p = thread + 256 u
// of the thread: (i, j) = (p % ka, p / ka), or the lower triangle by columns.
template <typename T, int U>
__global__ void __launch_bounds__(256) atb_packed_kernel(const T *__restrict__ A, int64_t lda, const T *__restrict__ B,
                                                         int64_t ldb, int64_t n, int ka, int kb,
                                                         int64_t rows_per_chunk, int symmetric, T *P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int sa_ld = ka | 1, sb_ld = kb | 1;  // odd: rows of a column fall on different banks
    T *sa = (T *)smem_raw, *sb = symmetric ? sa : sa + kAtbPackedRows * sa_ld;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int outputs = symmetric ? ka * (ka + 1) / 2 : ka * kb;
    int ia[U], ib[U];
    T acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int p = min(tid + 256 * u, outputs - 1);
        int i, j;
        if (symmetric) {  // column j of the lower triangle starts at j ka - j (j - 1) / 2
            j = (int)(((float)(2 * ka + 1) - sqrtf((float)(2 * ka + 1) * (2 * ka + 1) - 8.f * p)) * 0.5f);
            while (j > 0 && j * ka - j * (j - 1) / 2 > p) --j;
            while ((j + 1) * ka - (j + 1) * j / 2 <= p) ++j;
            i = j + p - (j * ka - j * (j - 1) / 2);
        } else {
            i = p % ka;
            j = p / ka;
        }
        ia[u] = i;
        ib[u] = j;
        acc[u] = T(0);
    }
    const int64_t r_beg = (int64_t)blockIdx.x * rows_per_chunk, r_end = min(r_beg + rows_per_chunk, n);
    for (int64_t r0 = r_beg; r0 < r_end; r0 += kAtbPackedRows) {
        const bool in = r0 + lane < r_end;  // columns are contiguous over rows: a lane per row
        for (int c = warp; c < ka; c += 8) sa[lane * sa_ld + c] = in ? A[r0 + lane + c * lda] : T(0);
        if (!symmetric)
            for (int c = warp; c < kb; c += 8) sb[lane * sb_ld + c] = in ? B[r0 + lane + c * ldb] : T(0);
        __syncthreads();
        const int ld2 = symmetric ? sa_ld : sb_ld;
#pragma unroll 4
        for (int r = 0; r < kAtbPackedRows; ++r)
#pragma unroll
            for (int u = 0; u < U; ++u) acc[u] = fma(sa[r * sa_ld + ia[u]], sb[r * ld2 + ib[u]], acc[u]);
        __syncthreads();
    }
    T *Pz = P + (int64_t)blockIdx.x * ka * kb;
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (tid + 256 * u < outputs) Pz[ia[u] + (int64_t)ib[u] * ka] = acc[u];
}

// Partial P[z] = A[rows of chunk z]^T B[rows of chunk z] for tile (I, J);
// symmetric (A == B): only tiles I >= J.  Thread (tx, ty) owns outputs
// (I*32 + ty + 8u, J*32 + tx), u < 4.
template <typename T>
__global__ void __launch_bounds__(256) atb_partial_kernel(const T *__restrict__ A, int64_t lda,
                                                          const T *__restrict__ B, int64_t ldb, int64_t n,
                                                          int64_t ka, int64_t kb, int64_t rows_per_chunk,
                                                          int symmetric, T *P) {
    const int I = blockIdx.y, J = blockIdx.z;
    if (symmetric && I < J) return;
    __shared__ T sa[kAtbTile][kAtbTile + 1], sb[kAtbTile][kAtbTile + 1];  // [row][column]
    const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;
    const int64_t r_beg = (int64_t)blockIdx.x * rows_per_chunk;
    const int64_t r_end = r_beg + rows_per_chunk < n ? r_beg + rows_per_chunk : n;
    T acc[4] = {T(0), T(0), T(0), T(0)};
    for (int64_t r0 = r_beg; r0 < r_end; r0 += kAtbTile) {
        // columns are contiguous over rows: lane tx walks the rows (coalesced)
        for (int c = ty; c < kAtbTile; c += 8) {
            const int64_t r = r0 + tx;
            const int64_t ca = (int64_t)I * kAtbTile + c, cb = (int64_t)J * kAtbTile + c;
            sa[tx][c] = (r < r_end && ca < ka) ? A[r + ca * lda] : T(0);
            sb[tx][c] = (r < r_end && cb < kb) ? B[r + cb * ldb] : T(0);
        }
        __syncthreads();
#pragma unroll 8
        for (int rr = 0; rr < kAtbTile; ++rr) {
            const T b = sb[rr][tx];
#pragma unroll
            for (int u = 0; u < 4; ++u) acc[u] = fma(sa[rr][ty + 8 * u], b, acc[u]);
        }
        __syncthreads();
    }
    T *Pz = P + (int64_t)blockIdx.x * ka * kb;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int64_t i = (int64_t)I * kAtbTile + ty + 8 * u, j = (int64_t)J * kAtbTile + tx;
        if (i < ka && j < kb) Pz[i + j * ka] = acc[u];
    }
}

// C[i, j] = sum over chunks of P[z][i, j], chunks g, g + 8, .. by thread group g and
// then the eight sums in order; symmetric: the upper part mirrors the lower.
template <typename T>
__global__ void __launch_bounds__(256) atb_reduce_kernel(const T *__restrict__ P, int64_t chunks, int64_t ka,
                                                         int64_t kb, int symmetric, T *C, int64_t ldc) {
    __shared__ T part[8][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int64_t e = (int64_t)blockIdx.x * 32 + lane;
    const int64_t i = e % ka, j = e / ka;
    T s = T(0);
    if (e < ka * kb) {
        const int64_t src = (symmetric && i < j) ? j + i * ka : e;
#pragma unroll 4
        for (int64_t z = g; z < chunks; z += 8) s += P[z * ka * kb + src];
    }
    part[g][lane] = s;
    __syncthreads();
    if (g == 0 && e < ka * kb) {
        for (int h = 1; h < 8; ++h) s += part[h][lane];
        C[i + j * ldc] = s;
    }
}

template <typename T>
int atb_launch(const T *A, int64_t lda, const T *B, int64_t ldb, int64_t n, int64_t ka, int64_t kb, T *C,
               int64_t ldc, T *P, int symmetric, cudaStream_t st) {
    if (ka == 0 || kb == 0) return 0;
    if (n == 0) return cudaMemsetAsync(P, 0, sizeof(T) * ka * kb, st) == cudaSuccess &&
                               cudaMemcpy2DAsync(C, sizeof(T) * ldc, P, sizeof(T) * ka, sizeof(T) * ka, kb,
                                                 cudaMemcpyDeviceToDevice, st) == cudaSuccess
                           ? 0
                           : -1;
    const int64_t chunks = atb_chunks(n, ka, kb, symmetric);
    const int64_t rpc = (n + chunks - 1) / chunks;
    if (atb_packed(ka, kb, symmetric)) {
        LaunchScope ls(K_MISC, st, 2.0 * n * ka * kb);
        const size_t smem = sizeof(T) * kAtbPackedRows * ((ka | 1) + (symmetric ? 0 : (kb | 1)));
        const int64_t u = (atb_outputs(ka, kb, symmetric) + 255) / 256;
        auto kern = u <= 1   ? atb_packed_kernel<T, 1>
                    : u <= 2 ? atb_packed_kernel<T, 2>
                    : u <= 4 ? atb_packed_kernel<T, 4>
                             : atb_packed_kernel<T, 8>;
        kern<<<(unsigned)chunks, 256, smem, st>>>(A, lda, B, ldb, n, (int)ka, (int)kb, rpc, symmetric, P);
        if (cudaGetLastError() != cudaSuccess) return -1;
    } else {
        const int64_t ti = (ka + kAtbTile - 1) / kAtbTile, tj = (kb + kAtbTile - 1) / kAtbTile;
        if (ti > 65535 || tj > 65535) return -1;
        LaunchScope ls(K_MISC, st, 2.0 * n * ka * kb);
        atb_partial_kernel<T><<<dim3((unsigned)chunks, (unsigned)ti, (unsigned)tj), 256, 0, st>>>(
            A, lda, B, ldb, n, ka, kb, rpc, symmetric, P);
        if (cudaGetLastError() != cudaSuccess) return -1;
    }
    LaunchScope ls(K_MISC, st, (double)chunks * ka * kb);
    atb_reduce_kernel<T><<<(unsigned)((ka * kb + 31) / 32), 256, 0, st>>>(P, chunks, ka, kb, symmetric, C, ldc);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// X (n x k, k <= KM) <- X L^-T for the lower k x k L: every row of X is a
// right-hand side of L z = x, solved by one thread in shared memory with the
// reference's sequence (src/triangular.rs:113-125: divide, subtract from all later
// entries; multiply and subtract rounded separately when EXACT).  The substitution
// kernel's one warp per right-hand side spends a warp instruction on a term of one
// of them; a lane each serves 32 (40000 x 20: 200 us and two transpositions ->
// 110 us).  A row in registers needs every loop unrolled, some 60 KB of code that
// each SM runs through a few times: it waited for instructions; a few rolled loops
// over shared memory take 46 us (the FP64 pipe's share is 38).
__device__ __noinline__ double rows_div_library(double a, double b) { return __ddiv_rn(a, b); }

template <typename T, bool kExact, int KM>
__global__ void __launch_bounds__(64) solve_rows_kernel(const T *__restrict__ L, int64_t ldl, int k, T *X, int64_t ldx,
                                                        int64_t n) {
    using Ar = Arith<T>;
    constexpr bool kInt = sizeof(T) == 8;  // FP64 quotients in integer arithmetic (lla_int_math.h)
    __shared__ T l[KM][KM];                // [column][row]
    __shared__ ImDivisor dq[kInt ? KM : 1];
    for (int e = threadIdx.x; e < KM * KM; e += blockDim.x) {
        const int r = e % KM, c = e / KM;
        l[c][r] = (r < k && c <= r) ? L[r + c * ldl] : T(0);
    }
    if (kInt && (int)threadIdx.x < k) dq[threadIdx.x] = im_divisor((double)L[threadIdx.x * (ldl + 1)]);
    __syncthreads();
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n) return;
    __shared__ T vs[KM][64];  // this thread's row: vs[.][threadIdx.x]
    T(*v)[64] = reinterpret_cast<T(*)[64]>(&vs[0][threadIdx.x]);
    bool ok = true;
    auto solve = [&](bool lib) {
#pragma unroll 4
        for (int c = 0; c < k; ++c) v[c][0] = X[row + c * ldx];
#pragma unroll 1
        for (int c = 0; c < k; ++c) {
            const T b = v[c][0];
            T x;
            if (kInt && !lib) {
                bool good;
                x = (T)im_div((double)b, dq[c], good);
                ok = ok && good;
            } else if (kInt) {
                x = (T)rows_div_library((double)b, (double)l[c][c]);
            } else {
                x = Ar::div(b, l[c][c]);
            }
            v[c][0] = x;
#pragma unroll 1
            for (int r = c + 1; r < k; r += 4) {
                T t[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) t[u] = r + u < k ? v[r + u][0] : T(0);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (r + u < k) t[u] = kExact ? Ar::sub(t[u], Ar::mul(x, l[c][r + u])) : Ar::fma_(-x, l[c][r + u], t[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (r + u < k) v[r + u][0] = t[u];
            }
        }
    };
    solve(false);
    if (!ok) solve(true);  // a quotient that the integer form does not take
#pragma unroll 4
    for (int c = 0; c < k; ++c) X[row + c * ldx] = v[c][0];
}

template <typename T>
int solve_rows_launch(const T *L, int64_t ldl, int64_t k, T *X, int64_t ldx, int64_t n, bool exact, cudaStream_t st) {
    if (n == 0 || k == 0) return 0;
    if (k > kSolveRowsMax) return -1;
    LaunchScope ls(K_TRSM, st, (double)k * k * n);
    auto kern = k <= 16   ? (exact ? solve_rows_kernel<T, true, 16> : solve_rows_kernel<T, false, 16>)
                : k <= 32 ? (exact ? solve_rows_kernel<T, true, 32> : solve_rows_kernel<T, false, 32>)
                          : (exact ? solve_rows_kernel<T, true, 48> : solve_rows_kernel<T, false, 48>);
    kern<<<(unsigned)((n + 63) / 64), 64, 0, st>>>(L, ldl, (int)k, X, ldx, n);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template int solve_rows_launch<double>(const double *, int64_t, int64_t, double *, int64_t, int64_t, bool,
                                       cudaStream_t);
template int solve_rows_launch<float>(const float *, int64_t, int64_t, float *, int64_t, int64_t, bool, cudaStream_t);

// V[r, c] -= sum_t Y[r, t] U[t, c]  (V n x k, Y n x ky, U ky x k; column-major)
template <typename T>
__global__ void __launch_bounds__(256) sub_tall_kernel(T *V, int64_t ldv, const T *__restrict__ Y, int64_t ldy,
                                                       const T *__restrict__ U, int64_t ldu, int64_t n,
                                                       int64_t ky) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (r >= n) return;
    T s = T(0);
    for (int64_t t = 0; t < ky; ++t) s = fma(Y[r + t * ldy], U[t + c * ldu], s);
    V[r + c * ldv] -= s;
}

template <typename T>
int sub_tall_launch(T *V, int64_t ldv, const T *Y, int64_t ldy, const T *U, int64_t ldu, int64_t n, int64_t ky,
                    int64_t k, cudaStream_t st) {
    if (n == 0 || k == 0 || ky == 0) return 0;
    if (k > 65535) return -1;
    LaunchScope ls(K_MISC, st, 2.0 * n * ky * k);
    sub_tall_kernel<T><<<dim3((unsigned)((n + 255) / 256), (unsigned)k), 256, 0, st>>>(V, ldv, Y, ldy, U, ldu, n,
                                                                                       ky);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template int atb_launch<double>(const double *, int64_t, const double *, int64_t, int64_t, int64_t, int64_t,
                                double *, int64_t, double *, int, cudaStream_t);
template int atb_launch<float>(const float *, int64_t, const float *, int64_t, int64_t, int64_t, int64_t,
                               float *, int64_t, float *, int, cudaStream_t);
template int sub_tall_launch<double>(double *, int64_t, const double *, int64_t, const double *, int64_t,
                                     int64_t, int64_t, int64_t, cudaStream_t);
template int sub_tall_launch<float>(float *, int64_t, const float *, int64_t, const float *, int64_t, int64_t,
                                    int64_t, int64_t, cudaStream_t);

}  // namespace lla
