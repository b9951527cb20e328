// lla_trsm.cu -- triangular solve op(T) X = B, in place on B (n x m), for a
// column-major triangular matrix M on the device.
//
// The reference's substitution (src/triangular.rs:113-125) walks the rows in
// "processing order" -- ascending for Lower, descending for Upper -- and, for
// each row i, divides b[i] by the diagonal and subtracts coeff * a[r, i] from
// every later row r.  Seen from one row r, that is
//     b[r] <- b[r] - x[i] * T[r, i]   for every earlier row i, in processing order,
//     x[r]  = b[r] / diag(r).
// This kernel keeps exactly that per-row sequence: row blocks of 32 are
// processed left-looking, each CTA applying the already-solved blocks in
// processing order and then solving its own diagonal block.  In EXACT mode
// every product and difference is rounded separately (b + (-c)*a equals
// b - c*a exactly in IEEE arithmetic), so X is bit-identical to the
// reference's; FAST mode uses FMA.
//
// Scheduling ("look-back"): each CTA takes a ticket from an atomic counter;
// tickets map to (row block, RHS chunk) in processing order, so a CTA only
// waits for row blocks whose CTAs took earlier tickets and are therefore
// already resident -- the wait always ends.  Every wait is bounded: after
// kSpinLimit polls the CTA records LLA_ERR_TIMEOUT in `err_word`, publishes
// its flag and returns, so a fault elsewhere cannot hang the device.
//
// What bounds it is the chain from row block to row block: hand-off, the last
// coupling tile, the solve of the diagonal block.  One warp owns one right-hand
// side of the block (lane = row) and goes from poll to publication alone; the
// CTA's warps share only the coupling tiles, copied one tile ahead into two
// buffers, and the diagonal block, which is loaded and prepared before the
// first wait.  An FP64 instruction takes 64 cycles of its sub-partition, so the
// solve of a block keeps few of them in its chain: in EXACT mode the division by
// the diagonal is done in integers, for FP32 by FMAs (lla_int_math.h); in FAST mode
// the rows are divided by their diagonal beforehand and a step is one FMA.  Four
// right-hand sides a CTA: one warp per sub-partition.
// Per row block: EXACT f64 9.9 us (n = 512; 25 with the library's division and the
// hand-over by the whole CTA), EXACT f32 2.9 (n = 1000, 8 right-hand sides; 7.1), FAST
// f64 7.3 (n = 8192, 16 right-hand sides; 30; 1.03 ms of the 1.9 ms solve is the FP64
// pipe's share), FAST f32 2.0 (n = 6001, 3 right-hand sides; 9.4).
//
// T[r, c] (logical) = trans ? M[c, r] : M[r, c]; `diag` (optional) overrides
// the diagonal as the reference's diag_fn does (src/triangular.rs:133-144).
#include <atomic>

#include "lla_common.cuh"
#include "lla_int_math.h"
#include "lla_kernels.h"
#include "lla_prof.h"

namespace lla {

constexpr int kTrsmNb = 32;
constexpr int kTrsmMaxMc = 8;
constexpr int kTrsmMc = 4;  // right-hand sides a CTA (8 where the flags would not fit otherwise)

__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void or_release(int *p, int v) {
    asm volatile("red.release.gpu.global.or.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <typename T>
__device__ __forceinline__ void cp_async_elem(T *dst, const T *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(sizeof(T))
                 : "memory");
}

// Warps of a CTA: one per right-hand side; at least four copy the tiles.
static int trsm_warps(int mc) { return std::max(mc, kTrsmMc); }

// The division of the reference's substitution by a divisor that is known early,
// without a test on its chain; ok says afterwards whether x is IEEE division's
// num / d, and the solve repeats a block with IEEE division if one was not (so does
// the FAST solve whose rows were divided beforehand, if a result is not finite).
// (EXACT f64 n = 512 165 us a solve, tested in every step 190; EXACT f32 n = 1000 99,
// tested in every step 137, with the general division 123.)
template <typename T>
struct TrsmDivisor;
template <>
struct TrsmDivisor<float> {
    FloatDivisor q;
    __device__ __forceinline__ explicit TrsmDivisor(float v) { q = float_divisor(v); }
    __device__ __forceinline__ float divide(float b) const { return float_div(b, q); }
    __device__ __forceinline__ bool ok(float num, float x) const { return float_div_ok(num, x, q); }
};
template <>
struct TrsmDivisor<double> {
    ImDivisor q;
    __device__ __forceinline__ explicit TrsmDivisor(double v) { q = im_divisor(v); }
    __device__ __forceinline__ double divide(double b) const {
        bool unused;
        return im_div(b, q, unused);
    }
    __device__ __forceinline__ bool ok(double num, double) const {
        bool good;
        im_div(num, q, good);
        return good;
    }
};

__device__ __forceinline__ bool trsm_finite(double v) { return ((unsigned)__double2hiint(v) & 0x7ff00000u) != 0x7ff00000u; }
__device__ __forceinline__ bool trsm_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }

// FAST, for a block that the products by reciprocals do not take: solved by division,
// from M itself.  Returns this lane's result.  Out of line with its addresses, and apart
// from the other form's repeat: sharing one repeat cost every block 2% (n = 2048, 16
// right-hand sides).
template <typename T>
__device__ __noinline__ T trsm_block_by_division(T bv, T dv, const T *M, int64_t ld, int64_t n, int lower, int trans,
                                                 int64_t t0, int bs) {
    using Ar = Arith<T>;
    const int tx = threadIdx.x;
    const int64_t step = lower ? 1 : -1, c0 = lower ? t0 : n - 1 - t0, r = c0 + step * tx;  // (rows in processing order)
    const T *const mrow = trans ? M + c0 + r * ld : M + r + c0 * ld;
    const int64_t mstep = trans ? step : step * ld;
#pragma unroll 1
    for (int y = 0; y < bs; ++y) {
        const T t = tx > y && tx < bs ? mrow[y * mstep] : T(0);
        const T xy = __shfl_sync(0xffffffffu, Ar::div(bv, dv), y);
        const T nb = Ar::fma_(-xy, t, bv);
        bv = tx == y ? xy : (tx > y ? nb : bv);
    }
    return bv;
}

template <typename T, bool kExact>
__global__ void __launch_bounds__(kTrsmNb *kTrsmMaxMc) trsm_lookback(const T *__restrict__ M, int64_t ld, int64_t n,
                                                                   int lower, int trans, const T *__restrict__ diag,
                                                                   T *B, int64_t ldb, int64_t m, int mc, int n_chunks,
                                                                   int *ws, int *err_word, int *sticky,
                                                                   long long spin_limit, int lose_first,
                                                                   const FactorVerdict *behind) {
    using Ar = Arith<T>;
    __shared__ T ts[2][kTrsmNb][kTrsmNb + 1];  // coupling tiles, [term][row]
    __shared__ T td[kTrsmNb][kTrsmNb + 1];     // diagonal block, [term][row]
    __shared__ __align__(16) T xs[kTrsmMaxMc][kTrsmNb];  // a solved block, by right-hand side
    __shared__ int s_ticket;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int tid = ty * kTrsmNb + tx, nthr = kTrsmNb * blockDim.y;
    int *counter = ws, *flags = ws + 1;
    // no ticket: the factorisation does not stand (the same for every CTA)
    if (tid == 0) s_ticket = behind != nullptr && !factor_stands(factor_verdict(behind)) ? -1 : atomicAdd(counter, 1);
    __syncthreads();
    if (s_ticket < 0) return;
    // failure injection (tests only): the first item is lost -- never solved,
    // never published -- so every wait on it runs out
    if (lose_first && s_ticket == 0) return;
    const int64_t rb = s_ticket / n_chunks;
    const int cc = s_ticket % n_chunks;
    const int64_t col = (int64_t)cc * mc + ty;
    const bool col_ok = ty < mc && col < m;  // uniform for the warp
    auto row_of = [&](int64_t t) -> int64_t { return lower ? t : n - 1 - t; };
    const int64_t t0 = rb * kTrsmNb;
    const int bs = (int)(n - t0 < kTrsmNb ? n - t0 : kTrsmNb);
    // element e of a tile: consecutive e -> consecutive memory (rows, or terms when transposed)
    auto copy_tile = [&](T(*dst)[kTrsmNb + 1], int64_t u0, int terms) {
        for (int e = tid; e < kTrsmNb * kTrsmNb; e += nthr) {
            const int x = trans ? e / kTrsmNb : e % kTrsmNb, y = trans ? e % kTrsmNb : e / kTrsmNb;
            if (x < bs && y < terms) {
                const int64_t r = row_of(t0 + x), c = row_of(u0 + y);
                cp_async_elem(&dst[y][x], trans ? &M[c + r * ld] : &M[r + c * ld]);
            } else {
                dst[y][x] = T(0);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    copy_tile(td, t0, bs);
    if (rb > 0) copy_tile(ts[0], 0, kTrsmNb);
    const int64_t r_own = row_of(t0 + (tx < bs ? tx : 0));
    T bv = (tx < bs && col_ok) ? B[r_own + col * ldb] : T(0);
    const T dv = tx < bs ? (diag ? diag[r_own] : M[r_own + r_own * ld]) : T(1);
    const TrsmDivisor<T> dq(dv);
    // FAST: 1 / dv in two parts, so that b times it is rounded once, like the quotient
    const T rinv = kExact ? T(0) : Ar::div(T(1), dv);
    const T rlo = kExact ? T(0) : Ar::mul(Ar::fma_(-dv, rinv, T(1)), rinv);
    if (rb > 0)
        asm volatile("cp.async.wait_group 1;" ::: "memory");
    else
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // FAST: the rows are divided by their diagonal, so that a step of the solve is
    // one FMA -- unless that would leave the comfortable range of the type (a zero,
    // tiny, huge or non-finite diagonal or entry): then a step divides.
    bool scaled = false;
    if (!kExact) {
        const T big = sizeof(T) == 8 ? T(1.3e154) : T(1.8e19f), small = T(1) / big;
        bool in_range = abs(rinv) <= big && abs(rinv) >= small;
        for (int y = ty; y < kTrsmNb; y += blockDim.y) {  // this lane's row
            const T t = abs(td[y][tx]), u = t * abs(rinv);
            in_range = in_range && (t == T(0) || y >= tx || (u <= big && u >= small));
        }
        scaled = __syncthreads_and(in_range) != 0;
        if (scaled)
            for (int y = ty; y < kTrsmNb; y += blockDim.y) td[y][tx] *= rinv;
    }

    bool abort = false;
    for (int64_t q = 0; q < rb; ++q) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        // tile q has landed for everyone, and tile q - 1's buffer is free; the barrier carries the
        // verdict of the last wait, so that all warps leave together
        if (__syncthreads_or(abort)) {
            abort = true;
            break;
        }
        if (q + 1 < rb) copy_tile(ts[(q + 1) & 1], (q + 1) * kTrsmNb, kTrsmNb);
        if (col_ok) {
            const int *f = flags + q * n_chunks + cc;
            long long spins = 0;
            while (!((ld_acquire(f) >> ty) & 1)) {
                if (*(volatile int *)err_word != 0) {
                    abort = true;
                    break;
                }
                if (++spins > spin_limit) {
                    if (tx == 0) {
                        atomicCAS(err_word, 0, (int)LLA_ERR_TIMEOUT);
                        if (sticky) atomicCAS(sticky, 0, (int)LLA_ERR_TIMEOUT);
                    }
                    abort = true;
                    break;
                }
                // only the block right before this one is worth polling without a pause: thousands of
                // warps wait further back, on the same few lines (n = 8192, 16 right-hand sides:
                // 1.98 ms a solve without the pause, 1.86 with it)
                if (q + 1 < rb) {
                    if (spins > 2) __nanosleep(256);
                } else if (spins > 64) {
                    __nanosleep(64);
                }
            }
            abort = __any_sync(0xffffffffu, abort);
            // solved block q (always a full block: q < rb), one row a lane
            __syncwarp();  // (the previous block's values have been read)
            xs[ty][tx] = abort ? T(0) : __ldcg(&B[row_of(q * kTrsmNb + tx) + col * ldb]);
            __syncwarp();
            const T(*tq)[kTrsmNb + 1] = ts[q & 1];
#pragma unroll
            for (int y0 = 0; y0 < kTrsmNb; y0 += 8) {
                T xv[8], tv[8];
#pragma unroll
                for (int y = 0; y < 8; ++y) {
                    xv[y] = xs[ty][y0 + y];
                    tv[y] = tq[y0 + y][tx];
                }
#pragma unroll
                for (int y = 0; y < 8; ++y)
                    bv = kExact ? Ar::sub(bv, Ar::mul(xv[y], tv[y])) : Ar::fma_(-xv[y], tv[y], bv);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!kExact) __syncthreads();  // (the first block met no barrier after the scaling of td)

    if (!abort && col_ok) {
        if (scaled) {
            const T b0 = bv;
            bv = Ar::fma_(bv, rinv, Ar::mul(bv, rlo));
#pragma unroll 4
            for (int y = 0; y < bs; ++y) {
                const T xy = __shfl_sync(0xffffffffu, bv, y);
                const T nb = Ar::fma_(-xy, td[y][tx], bv);
                if (tx > y) bv = nb;
            }
            // infinities and overflow on the way: products by a reciprocal are no longer what the
            // division gives (inf * 0, inf - inf)
            if (!__all_sync(0xffffffffu, tx >= bs || trsm_finite(bv))) {
                bv = trsm_block_by_division<T>(b0, dv, M, ld, n, lower, trans, t0, bs);
            }
        } else {
            const T b0 = bv;
            T num = bv;  // what this lane's row was divided from
#pragma unroll 4
            for (int y = 0; y < bs; ++y) {
                const T xy = __shfl_sync(0xffffffffu, dq.divide(bv), y);  // coeff = b[i,k] / diag  (:117-119)
                const T nb = kExact ? Ar::sub(bv, Ar::mul(xy, td[y][tx])) : Ar::fma_(-xy, td[y][tx], bv);
                num = tx == y ? bv : num;
                bv = tx == y ? xy : (tx > y ? nb : bv);
            }
            const bool ok = tx >= bs || dq.ok(num, bv);
            if (!__all_sync(0xffffffffu, ok)) {
                bv = b0;
#pragma unroll 1
                for (int y = 0; y < bs; ++y) {
                    const T xy = __shfl_sync(0xffffffffu, Ar::div(bv, dv), y);
                    const T nb = kExact ? Ar::sub(bv, Ar::mul(xy, td[y][tx])) : Ar::fma_(-xy, td[y][tx], bv);
                    bv = tx == y ? xy : (tx > y ? nb : bv);
                }
            }
        }
    }
    if (tx < bs && col_ok) B[r_own + col * ldb] = bv;
    __syncwarp();  // the warp's stores, then its bit of the block's flag
    if (tx == 0) or_release(flags + rb * n_chunks + cc, 1 << ty);
}

// One-shot failure injection for the tests of timeout reporting
// (lla_debug_inject_lost_handoff): the next triangular-solve launch loses its
// first item and its waits give up after the armed number of polls.
static std::atomic<long long> g_inject_spin{-1};  // -1: nothing armed

struct TrsmWaitCfg {
    long long spin_limit;
    int lose_first;
};

static TrsmWaitCfg take_wait_cfg() {
    const long long s = g_inject_spin.exchange(-1);
    if (s < 0) return {kSpinLimit, 0};
    return {s > 0 ? s : kSpinLimit, 1};
}

template <typename T>
int trsm_launch(const T *M, int64_t ld, int64_t n, int lower, int trans, const T *diag, T *B,
                int64_t ldb, int64_t m, bool exact, int *ws, int *err_word, cudaStream_t st,
                int *sticky, const FactorVerdict *behind) {
    if (n == 0 || m == 0) return 0;
    const int mc = (int)std::min<int64_t>(kTrsmMc, m);
    const int64_t chunks = ceil_div(m, mc);
    const int64_t R = ceil_div(n, kTrsmNb);
    if (cudaMemsetAsync(ws, 0, sizeof(int) * (1 + R * chunks), st) != cudaSuccess) return -1;
    const dim3 block(kTrsmNb, trsm_warps(mc));
    const unsigned grid = (unsigned)(R * chunks);
    const TrsmWaitCfg wc = take_wait_cfg();
    // algorithmic work: n^2 * m flops (n(n-1)/2 multiply-adds and n divisions per column)
    LaunchScope ls(K_TRSM, st, (double)n * n * m);
    if (exact)
        trsm_lookback<T, true><<<grid, block, 0, st>>>(M, ld, n, lower, trans, diag, B, ldb, m, mc,
                                                       (int)chunks, ws, err_word, sticky,
                                                       wc.spin_limit, wc.lose_first, behind);
    else
        trsm_lookback<T, false><<<grid, block, 0, st>>>(M, ld, n, lower, trans, diag, B, ldb, m,
                                                        mc, (int)chunks, ws, err_word, sticky,
                                                        wc.spin_limit, wc.lose_first, behind);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

size_t trsm_ws_ints(int64_t n, int64_t m) {
    if (n == 0 || m == 0) return 1;
    const int mc = (int)std::min<int64_t>(kTrsmMc, m);
    return (size_t)(1 + ceil_div(n, kTrsmNb) * ceil_div(m, mc));
}

template int trsm_launch<double>(const double *, int64_t, int64_t, int, int, const double *, double *, int64_t,
                                 int64_t, bool, int *, int *, cudaStream_t, int *, const FactorVerdict *);
template int trsm_launch<float>(const float *, int64_t, int64_t, int, int, const float *, float *, int64_t,
                                int64_t, bool, int *, int *, cudaStream_t, int *, const FactorVerdict *);

}  // namespace lla

// ---------------------------------------------------------------------------
// Allocation-free triangular solve (lla_dtrsm_device_noalloc).
//
// Some callers cannot call cudaMalloc: code that runs inside another
// library's memory-pool callback, processes whose device memory is carved up
// once at start-up by a host framework that owns every allocation, or
// latency-critical loops where an allocation would synchronise the device.
// This entry point takes its ticket/flag scratch from a fixed, file-scope
// device array instead of library-owned buffers.  The array is part of the
// module image, so every GPU that loads the library holds it (a little over
// 256 KiB) until the process exits.
//
// Host code cannot use the array's name as a device address (on the host it
// names a stand-in object); the device address is obtained once per device
// with cudaGetSymbolAddress, on the first call made while that device is
// current, and cached.  That first call therefore also does the set-up and
// should come before any stream capture.  The cache is not refreshed after a
// cudaDeviceReset (which unloads the module), so the entry point must not be
// used across a device reset.
//
// All calls share the one array and it keeps the last call's contents: each
// call clears the part it uses before its launch, and calls whose work
// overlaps on the GPU (different streams, or different host threads without
// ordering) race on it.  A bounded wait that gives up is recorded in the
// array's status word, which lla_dtrsm_device_noalloc_status reads and clears.

#include <mutex>

namespace lla {

constexpr int kNoAllocMaxFlags = 1 << 16;  // row blocks x RHS chunks
constexpr int kNoAllocMaxDevices = 64;
// [0] ticket counter, [1 .. kNoAllocMaxFlags] flags, [kNoAllocMaxFlags + 1]
// error word of the current call, [kNoAllocMaxFlags + 2] status word (kept
// until lla_dtrsm_device_noalloc_status clears it)
constexpr int kNoAllocErr = kNoAllocMaxFlags + 1, kNoAllocStatus = kNoAllocMaxFlags + 2;
static __device__ __align__(256) int g_trsm_noalloc_scratch[kNoAllocMaxFlags + 3];

static std::mutex g_noalloc_mu;
static int *g_noalloc_addr[kNoAllocMaxDevices] = {};

static cudaError_t noalloc_scratch(int **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kNoAllocMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_trsm_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_addr[dev] = (int *)p;
    }
    *out = g_noalloc_addr[dev];
    return cudaSuccess;
}

}  // namespace lla

extern "C" int lla_dtrsm_device_noalloc(const double *dL, int64_t n, int64_t ld, int trans,
                                        double *dB, int64_t m, int64_t ldb, int algo, void *stream,
                                        lla_error *err) {
    using namespace lla;
    if (n < 0 || m < 0 || ld < std::max<int64_t>(1, n) || ldb < std::max<int64_t>(1, n) ||
        (n > 0 && m > 0 && (!dL || !dB)) || (algo != LLA_ALGO_EXACT && algo != LLA_ALGO_FAST))
        return lla__set_status(err, LLA_ERR_INVALID_ARG);
    lla__set_status(err, LLA_OK);
    if (n == 0 || m == 0) return LLA_OK;
    // the limit is that of eight right-hand sides a CTA; fewer where their flags fit too
    const int64_t R = ceil_div(n, kTrsmNb);
    const int mc = (int)std::min<int64_t>(R * ceil_div(m, kTrsmMc) <= kNoAllocMaxFlags ? kTrsmMc : kTrsmMaxMc, m);
    const int64_t chunks = ceil_div(m, mc);
    if (R * chunks > kNoAllocMaxFlags) return lla__set_status(err, LLA_ERR_TOO_LARGE);
    int *scratch = nullptr;
    cudaError_t e = noalloc_scratch(&scratch);
    if (e != cudaSuccess) return lla__set_cuda_error(err, e);
    cudaStream_t st = (cudaStream_t)stream;
    int *err_word = scratch + kNoAllocErr;
    e = cudaMemsetAsync(scratch, 0, sizeof(int) * (size_t)(1 + R * chunks), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(err_word, 0, sizeof(int), st);
    if (e != cudaSuccess) return lla__set_cuda_error(err, e);
    const dim3 block(kTrsmNb, trsm_warps(mc));
    const unsigned grid = (unsigned)(R * chunks);
    // trans = 0: L X = B (lower, ascending); trans = 1: L^T X = B (descending)
    const int lower = trans ? 0 : 1;
    const TrsmWaitCfg wc = take_wait_cfg();
    {
        // counted and timed like the allocating entry point's launches
        LaunchScope ls(K_TRSM, st, (double)n * n * m);
        if (algo == LLA_ALGO_EXACT)
            trsm_lookback<double, true><<<grid, block, 0, st>>>(
                dL, ld, n, lower, trans ? 1 : 0, nullptr, dB, ldb, m, mc, (int)chunks, scratch, err_word,
                scratch + kNoAllocStatus, wc.spin_limit, wc.lose_first, nullptr);
        else
            trsm_lookback<double, false><<<grid, block, 0, st>>>(
                dL, ld, n, lower, trans ? 1 : 0, nullptr, dB, ldb, m, mc, (int)chunks, scratch, err_word,
                scratch + kNoAllocStatus, wc.spin_limit, wc.lose_first, nullptr);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return lla__set_cuda_error(err, e);
    return LLA_OK;
}

// Synchronises `stream`, reads the status word that the allocation-free
// solves on the current device share, and clears it.  Allocates nothing.
extern "C" int lla_dtrsm_device_noalloc_status(void *stream, lla_error *err) {
    using namespace lla;
    lla__set_status(err, LLA_OK);
    int *scratch = nullptr;
    cudaError_t e = noalloc_scratch(&scratch);
    if (e != cudaSuccess) return lla__set_cuda_error(err, e);
    cudaStream_t st = (cudaStream_t)stream;
    int word = 0;
    e = cudaStreamSynchronize(st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&word, scratch + kNoAllocStatus, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && word != 0) e = cudaMemsetAsync(scratch + kNoAllocStatus, 0, sizeof(int), st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return lla__set_cuda_error(err, e);
    return word ? lla__set_status(err, word) : LLA_OK;
}

// Arms the one-shot failure injection of the next triangular-solve launch
// (tests of timeout reporting only).
extern "C" int lla_debug_inject_lost_handoff(int64_t spin_limit) {
    if (spin_limit < 0) return LLA_ERR_INVALID_ARG;
    lla::g_inject_spin.store((long long)spin_limit);
    return LLA_OK;
}
