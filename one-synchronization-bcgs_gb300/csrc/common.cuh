// Shared definitions for the GB300 BCGS kernels.
//
// Layout conventions (the reference's, include/orth.h): every tall matrix is
// column-major FP64 with a leading dimension `ld` >= rows; element (r, c) lives at
// p[r + c * ld]. Column offsets are always formed in 64-bit arithmetic (the
// reference forms them in `int`, SRC/orth.c:174,183,207, which overflows at
// m * n >= 2^31).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace bcgs {

using i64 = long long;

// Number of SMs on GB300; grids are sized in multiples of it.
constexpr int kNumSMsDefault = 152;

// Status word layout (device-resident, int32 each), read back by the host API.
//   [0] first Cholesky breakdown: 1-based block step, 0 if none
//   [1] dpotrf-style info of that breakdown (1-based column)
//   [2] bounded-wait timeout flag (reserved; no kernel here spins on a peer)
//   [3] internal argument error flag
constexpr int kStatusWords = 4;

__host__ __device__ inline i64 ceil_div(i64 a, i64 b) { return (a + b - 1) / b; }

// Chained launches. A block step is a chain of short kernels, each of which needs the
// whole one before it; launched plainly, every link costs the drain of one grid plus
// the start of the next, about 2 us. launch_chained lets the next grid be set up on the
// SMs while this one runs (programmatic stream serialization). Each kernel so launched
// starts with chain_enter: it waits until the grids before it in the stream have
// completed and their writes are visible, and then lets its own successor be set up, so
// that at most one grid waits at a time. So begins every kernel that launch_chained or
// launch_spread may launch; the others (batched, metrics, diagnostics) are launched plainly
// and neither start early nor let their successors.
#ifdef __CUDACC__
__device__ __forceinline__ void chain_enter() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... Params, class... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                  Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// The same for the kernels bound by the FP64 pipe, chained only while they have at most
// one CTA per SM. Their time is that of the SM with the most CTAs, and CTAs that are
// placed while the grid before still holds its SMs crowd onto the SMs that free up
// first: chained at any size, BCGSI+ at m = 10^5 took 31.4 instead of 24.7 ms and bcgsi2P2s
// at 4 10^5 x 32 39.0 instead of 22.1 ms.
template <class... Params, class... Args>
inline cudaError_t launch_spread(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                 Args&&... args) {
    if ((i64)grid.x * grid.y * grid.z <= kNumSMsDefault)
        return launch_chained(kernel, grid, block, smem, st, static_cast<Args&&>(args)...);
    kernel<<<grid, block, smem, st>>>(static_cast<Params>(args)...);
    return cudaPeekAtLastError();
}

// 1 / x for a normal x whose reciprocal is normal: one step of the third-order iteration
// for the zero of 1/r - x (Chebyshev's; J. F. Traub, Iterative Methods for the Solution of
// Equations, 1964), r (1 + e + e^2) with e = 1 - x r, from the hardware's approximate
// reciprocal (rcp.approx.ftz.f64). It leaves a relative error of e^3 and the roundings: with
// 19 bits or more in the first r, the result is within one unit in the last place of the
// division's. Three dependent operations, where a division takes 570 clocks.
__device__ __forceinline__ double recip(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// sqrt(d) from v = rsqrt(d), for a d of ordinary size: Newton's (Heron's) step for u^2 = d from
// u = d v, with v / 2 for 1 / (2 u). Within one unit in the last place of sqrt's, half the
// cost of a square root and a division where 1 / sqrt(d) is wanted too.
__device__ __forceinline__ double root(double d, double v) {
    const double u = d * v;
    return fma(fma(-u, u, d), 0.5 * v, u);
}

// Asynchronous copy of one double into shared memory; zero if not valid (src then only has to be
// readable).
__device__ __forceinline__ void cp_async8(double* dst, const double* src, bool valid) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
#endif

}  // namespace bcgs

#define BCGS_CUDA_TRY(expr)                                          \
    do {                                                             \
        cudaError_t _e = (expr);                                     \
        if (_e != cudaSuccess) return (int)_e;                       \
    } while (0)
