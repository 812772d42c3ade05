// Plain-FP64 update of the BCGS hot path (kernels; instantiated by update_fp64.cu and
// update_split_fp64.cu):
//   update_fp64 : Xc = (Xc - X[:, 0:K] S) T^{-1}, T upper triangular
// replaces dgemm('N','N') + dtrsm('R','U','N','N') (SRC/orth.c:173-176).
//
// One row per lane with NC register accumulators: S staged through shared memory, the
// right triangular scaling by forward substitution in registers, so the reference's
// dgemm and dtrsm are one pass. Bound by the FP64 pipe: an instruction of one warp takes
// its quarter of the SM for 64 clocks, so the time is K NC + NC^2 / 2 instructions per 32
// rows, on the SM quarter that has the most of them. Hence
//   * there is code for every width up to 16, every fourth to 32 and every eighth beyond (10
//     columns in 16 accumulators cost 60 % more);
//   * up to kSplitRows rows the warps of a CTA share 32 rows and split K four ways
//     (SPLIT), because 32-row units of the whole K are too coarse for the 608 SM
//     quarters: 10^5 rows are 5.1 units each, so some do 6.
// m = 10^5, n = 200, s = 10, 38 updates: 12.7 ms with 16 accumulators and 128 rows per
// CTA, 7.2 ms now (6.3 ms at the FP64 peak).
#pragma once

#include "batched.h"
#include "common.cuh"
#include "kernels.h"

namespace bcgs {

namespace {
constexpr int UP_THREADS = 128;
constexpr int UP_KCH = 64;                 // rows of S staged at a time (16 per warp if split)
constexpr i64 kSplitRows = 600000;         // 31 units of 32 rows per SM quarter: an uneven last one costs 3 %
constexpr int kSplitK = 32;                // the four partial sums cost 3 additions per output

template <int NC>
__host__ __device__ constexpr int up_kch() { return NC <= 16 ? UP_KCH : (NC <= 32 ? UP_KCH / 2 : UP_KCH / 4); }
// Shared-memory doubles: S chunk (or the three other warps' sums), T, T's reciprocal diagonal.
template <int NC, bool SPLIT>
__host__ __device__ constexpr int up_smem() {
    return (SPLIT && 3 * 32 > up_kch<NC>() ? 3 * 32 : up_kch<NC>()) * NC + NC * NC + NC;
}
inline bool up_split(i64 m, int K) { return m <= kSplitRows && K >= kSplitK; }
}  // namespace

// Rows [blk * 128, ...) of the update, one per thread, or with SPLIT rows [blk * 32, ...),
// each K summed in four quarters by the CTA's four warps and the quarters added in
// order. sm holds up_smem<NC, SPLIT>() doubles. Every sum is an FMA chain over its k in
// order, then the forward substitution in column order, so the result does not depend
// on NC >= nc.
template <int NC, bool SPLIT>
__device__ __forceinline__ void update_body(double* __restrict__ X, i64 ld, i64 m, int q0, int K, int c0, int nc,
                                            const double* __restrict__ S, int lds, const double* __restrict__ T,
                                            int ldt, i64 blk, double* __restrict__ sm) {
    constexpr int KCH = up_kch<NC>();
    constexpr int KW = SPLIT ? KCH / 4 : KCH;   // rows of the chunk a warp uses
    constexpr int UQ = NC <= 8 ? 8 : (NC <= 16 ? 4 : 2);   // loads in flight, NC 64 clocks of work each
    constexpr int SROWS = SPLIT && 3 * 32 > KCH ? 3 * 32 : KCH;
    double* sS = sm;
    double* sT = sm + SROWS * NC;
    double* sRd = sT + NC * NC;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const i64 r = SPLIT ? blk * 32 + lane : blk * UP_THREADS + tid;
    // The warp that finishes the rows: its substitution is the CTA's serial part, so it
    // falls on another SM quarter in each CTA.
    const int last = SPLIT ? (int)(blk & 3) : warp;
    if (T != nullptr) {
        for (int e = tid; e < NC * NC; e += UP_THREADS) {
            int i = e % NC, j = e / NC;
            sT[i * NC + j] = (i < nc && j < nc && i <= j) ? T[i + (i64)j * ldt] : 0.0;
        }
        __syncthreads();
        if (tid < NC) sRd[tid] = (tid < nc) ? 1.0 / sT[tid * NC + tid] : 0.0;
    }
    double acc[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) acc[j] = 0.0;
    const bool live = r < m;
    const int Kq = SPLIT ? (K + 3) / 4 : K;      // this warp's share [kw, kw + kn) of K
    const int kw = SPLIT ? min(K, warp * Kq) : 0, kn = SPLIT ? min(K, kw + Kq) - kw : K;
    for (int k0 = 0; k0 < Kq; k0 += KW) {
        __syncthreads();
        for (int e = tid; e < KCH * NC; e += UP_THREADS) {
            const int kk = e % KCH, j = e / KCH;
            const int k = SPLIT ? (kk / KW) * Kq + k0 + kk % KW : k0 + kk;
            const bool ok = j < nc && k < K && (!SPLIT || k0 + kk % KW < Kq);
            sS[kk * NC + j] = ok ? S[k + (i64)j * lds] : 0.0;
        }
        __syncthreads();
        const int kc = min(KW, kn - k0);
        if (live) {
            const double* qrow = X + r + (i64)(q0 + kw + k0) * ld;
            const double* sw = sS + (SPLIT ? warp * KW * NC : 0);
            int kk = 0;
            for (; kk + UQ <= kc; kk += UQ) {
                double q[UQ];
#pragma unroll
                for (int u = 0; u < UQ; ++u) q[u] = qrow[(i64)(kk + u) * ld];
#pragma unroll
                for (int u = 0; u < UQ; ++u)
#pragma unroll
                    for (int j = 0; j < NC; ++j) acc[j] = fma(q[u], sw[(kk + u) * NC + j], acc[j]);
            }
#pragma unroll 1
            for (; kk < kc; ++kk) {
                const double q = qrow[(i64)kk * ld];
#pragma unroll
                for (int j = 0; j < NC; ++j) acc[j] = fma(q, sw[kk * NC + j], acc[j]);
            }
        }
    }
    __syncthreads();
    if constexpr (SPLIT) {
        // Quarters 1 .. 3 go through shared memory, quarter 0 first in the sum; the warp
        // that adds them takes the others' from there.
        if (warp != last) {
            double* p = sS + ((warp - last + 4) % 4 - 1) * 32 * NC + lane;
#pragma unroll
            for (int j = 0; j < NC; ++j) p[j * 32] = acc[j];
        }
        __syncthreads();
        if (warp != last) return;
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            double v = 0.0;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const double x = w == last ? acc[j] : sS[((w - last + 4) % 4 - 1) * 32 * NC + j * 32 + lane];
                v = w == 0 ? x : v + x;
            }
            acc[j] = v;
        }
    }
    if (!live) return;   // no barrier follows
    double* xr = X + r + (i64)c0 * ld;
    // acc becomes w = x - Q S in place.
#pragma unroll
    for (int j = 0; j < NC; ++j) acc[j] = (j < nc) ? xr[(i64)j * ld] - acc[j] : 0.0;
    if (T != nullptr) {
        // Forward substitution u T = w (dtrsm 'R','U','N','N'), column by column.
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            double v = acc[j];
#pragma unroll
            for (int i = 0; i < j; ++i) v = fma(-acc[i], sT[i * NC + j], v);
            acc[j] = v * sRd[j];
        }
    }
#pragma unroll
    for (int j = 0; j < NC; ++j)
        if (j < nc) xr[(i64)j * ld] = acc[j];
}

template <int NC, bool SPLIT>
__global__ void __launch_bounds__(UP_THREADS)
update_fp64(double* __restrict__ X, i64 ld, i64 m, int q0, int K, int c0, int nc,
            const double* __restrict__ S, int lds, const double* __restrict__ T, int ldt,
            const int* __restrict__ gate) {
    __shared__ double sm[up_smem<NC, SPLIT>()];
    chain_enter();
    if (gate != nullptr && *gate == 0) return;
    update_body<NC, SPLIT>(X, ld, m, q0, K, c0, nc, S, lds, T, ldt, blockIdx.x, sm);
}

// The kernel for width nc (64 or less; 32 or less if SPLIT), launched over m rows.
template <bool SPLIT>
int launch_update_width(double* X, i64 ld, i64 m, int q0, int K, int c0, int nc, const double* S, int lds,
                        const double* T, int ldt, const int* gate, cudaStream_t st) {
    const unsigned grid = (unsigned)ceil_div(m, SPLIT ? 32 : UP_THREADS);
#define BCGS_UPD(N)                                                                                        \
    if (nc <= N) {                                                                                         \
        launch_spread(update_fp64<N, SPLIT>, grid, UP_THREADS, 0, st, X, ld, m, q0, K, c0, nc, S, lds, T, ldt, gate);    \
        break;                                                                                             \
    }
    do {
        BCGS_UPD(1) BCGS_UPD(2) BCGS_UPD(3) BCGS_UPD(4) BCGS_UPD(5) BCGS_UPD(6) BCGS_UPD(7) BCGS_UPD(8) BCGS_UPD(9)
        BCGS_UPD(10) BCGS_UPD(11) BCGS_UPD(12) BCGS_UPD(13) BCGS_UPD(14) BCGS_UPD(15) BCGS_UPD(16) BCGS_UPD(20)
        BCGS_UPD(24) BCGS_UPD(28) BCGS_UPD(32)
        if constexpr (!SPLIT) { BCGS_UPD(40) BCGS_UPD(48) BCGS_UPD(56) BCGS_UPD(64) }
        return (int)cudaErrorInvalidValue;
    } while (0);
#undef BCGS_UPD
    g_launch_count += 1;
    return (int)cudaGetLastError();
}
int launch_update_split_k(double* X, i64 ld, i64 m, int q0, int K, int c0, int nc, const double* S, int lds,
                          const double* T, int ldt, const int* gate, cudaStream_t st);

}  // namespace bcgs
