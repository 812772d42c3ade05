// Upper Gram of a narrow panel (nc <= 16 columns), for the checked Cholesky QR of TSQR panels.
//
// The general Gram's tiles pad 10 x 10 entries, of which 55 are wanted, to 16 x 16. Here a
// lane holds a row of the panel and all the wanted sums (up to 11 columns) or those of
// some of the columns (two warps share the rows beyond), so a row of 32 lanes takes
// nc (nc + 1) / 2 FP64 instructions and nothing is padded: 22 us at 10^5 x 10, 181 us at
// 7 10^5 x 16 (150 us at the FP64 peak).
// The lanes' sums are added through shared memory once per CTA, the CTAs' by the sliced
// reduction, all in a fixed order.
#include "common.cuh"
#include "kernels.h"

namespace bcgs {

namespace {
constexpr int PG_THREADS = 128;
constexpr int PG_CTAS_PER_SM = 3;

// Columns [0, pg_cut) go to the first warp of a pair, the rest to the second.
template <int NC>
__host__ __device__ constexpr int pg_cut() {
    return NC <= 11 ? NC : (NC * 7 + 5) / 10;   // about half of the sums
}
template <int NC>
__host__ __device__ constexpr int pg_slots() { return NC <= 11 ? 4 : 2; }   // row groups of 32 a CTA takes at once
template <int NC>
__host__ __device__ constexpr int pg_sums() { return NC * (NC + 1) / 2; }
template <int NC>
__host__ __device__ constexpr int pg_ld() { return 32 * pg_slots<NC>() + 1; }

// Columns [J0, J1) of the upper Gram over this warp's row groups, into red[sum][lane slot].
template <int NC, int J0, int J1>
__device__ __forceinline__ void panel_sums(const double* __restrict__ V, i64 ld, i64 m, int nc, i64 g0, i64 step,
                                           double* __restrict__ red, int col) {
    constexpr int NA = J1 * (J1 + 1) / 2 - J0 * (J0 + 1) / 2;
    double acc[NA], x[J1];
#pragma unroll
    for (int k = 0; k < NA; ++k) acc[k] = 0.0;
    const i64 groups = (m + 31) / 32;
    for (i64 g = g0; g < groups; g += step) {
        const i64 r = g * 32 + (threadIdx.x & 31);
#pragma unroll
        for (int c = 0; c < J1; ++c) x[c] = c < nc && r < m ? V[r + (i64)c * ld] : 0.0;
        int k = 0;
#pragma unroll
        for (int j = J0; j < J1; ++j)
#pragma unroll
            for (int i = 0; i <= j; ++i, ++k) acc[k] = fma(x[i], x[j], acc[k]);
    }
#pragma unroll
    for (int k = 0; k < NA; ++k) red[(J0 * (J0 + 1) / 2 + k) * pg_ld<NC>() + col] = acc[k];
}

template <int NC>
__global__ void __launch_bounds__(PG_THREADS)
panel_gram_kernel(const double* __restrict__ V, i64 ld, i64 m, int nc, double* __restrict__ part,
                  const int* __restrict__ gate) {
    extern __shared__ double red[];   // sums x lane slots, then 4 x sums
    chain_enter();
    if (gate != nullptr && *gate == 0) return;
    constexpr int SL = pg_slots<NC>(), NS = pg_sums<NC>(), LD = pg_ld<NC>(), CUT = pg_cut<NC>();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp % SL;
    const i64 g0 = (i64)blockIdx.x * SL + slot, step = (i64)gridDim.x * SL;
    if constexpr (CUT == NC) {
        panel_sums<NC, 0, NC>(V, ld, m, nc, g0, step, red, slot * 32 + lane);
    } else {
        if (warp < SL) panel_sums<NC, 0, CUT>(V, ld, m, nc, g0, step, red, slot * 32 + lane);
        else panel_sums<NC, CUT, NC>(V, ld, m, nc, g0, step, red, slot * 32 + lane);
    }
    __syncthreads();
    // Warp w adds the w-th quarter of the lane slots of every sum.
    double* quarter = red + NS * LD;
    for (int o = lane; o < NS; o += 32) {
        double s = 0.0;
#pragma unroll 8
        for (int k = 0; k < 8 * SL; ++k) s += red[o * LD + warp * 8 * SL + k];
        quarter[warp * NS + o] = s;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < NS; o += PG_THREADS) {
        int j = 0;
        while ((j + 1) * (j + 2) / 2 <= o) ++j;
        const int i = o - j * (j + 1) / 2;
        if (j < nc)
            part[(i64)blockIdx.x * nc * nc + i + (i64)j * nc] =
                (quarter[o] + quarter[NS + o]) + (quarter[2 * NS + o] + quarter[3 * NS + o]);
    }
}

// At least four row groups per warp, at most PG_CTAS_PER_SM CTAs per SM.
int panel_ctas(i64 m, int slots, int num_sms) {
    const i64 want = ceil_div(ceil_div(m, 32), 4 * slots), most = (i64)PG_CTAS_PER_SM * num_sms;
    return (int)(want < most ? want : most);
}

template <int NC>
int run_panel(const double* V, i64 ld, i64 m, int nc, double* G, double* part, int num_sms, const int* gate,
              cudaStream_t st) {
    const size_t smem = (size_t)(pg_sums<NC>() * (pg_ld<NC>() + 4)) * sizeof(double);
    int rc = smem_attr((const void*)panel_gram_kernel<NC>, (int)smem);
    if (rc) return rc;
    const int ctas = panel_ctas(m, pg_slots<NC>(), num_sms);
    launch_spread(panel_gram_kernel<NC>, (unsigned)ctas, PG_THREADS, smem, st, V, ld, m, nc, part, gate);
    g_launch_count += 1;
    rc = (int)cudaGetLastError();
    return rc ? rc : launch_gram_reduce_sliced(part, ctas, nc, nc, G, nc, false, st);
}
}  // namespace

i64 panel_gram_part_doubles(int nc) { return (i64)PG_CTAS_PER_SM * kNumSMsDefault * nc * nc; }

int launch_panel_gram(const double* X, i64 ld, i64 m, int c0, int nc, double* G, double* part, int num_sms,
                      const int* gate, cudaStream_t st) {
    const double* V = X + (i64)c0 * ld;
    if (num_sms > kNumSMsDefault) num_sms = kNumSMsDefault;   // part's size
    if (nc <= 8) return run_panel<8>(V, ld, m, nc, G, part, num_sms, gate, st);
    if (nc <= 10) return run_panel<10>(V, ld, m, nc, G, part, num_sms, gate, st);
    if (nc <= 12) return run_panel<12>(V, ld, m, nc, G, part, num_sms, gate, st);
    if (nc <= 14) return run_panel<14>(V, ld, m, nc, G, part, num_sms, gate, st);
    if (nc <= 16) return run_panel<16>(V, ld, m, nc, G, part, num_sms, gate, st);
    return (int)cudaErrorInvalidValue;
}

}  // namespace bcgs
