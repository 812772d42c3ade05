// Upper Gram of a narrow panel (nc <= 32 columns), for the checked Cholesky QR of TSQR panels.
//
// The general Gram's tiles pad 10 x 10 entries, of which 55 are wanted, to 16 x 16, and run
// three of four 16 x 16 tiles for 32 columns, 768 products for 528. Here a lane holds a
// row of the panel and all the wanted sums (up to 11 columns) or those of some of the
// columns (2, 4 or 8 warps share the rows beyond), so a row of 32 lanes takes
// nc (nc + 1) / 2 FP64 instructions and nothing is padded: 22 us at 10^5 x 10, 181 us at
// 7 10^5 x 16 (150 us at the FP64 peak), 416 us at 4 10^5 x 32 (335 us at the peak).
// Up to 16 columns three CTAs share an SM and hide each other's loads. Beyond, the sums
// fill the registers of one or two CTAs, so the rows come through a ring of stages in
// shared memory, each warp copying its own columns: bcgsi2P2s at 400000 x 256, s = 32,
// takes 22.3 ms with the general Gram, 20.4 ms with this one and loads straight into
// registers, 20.9 ms with prefetches too (they spill), 19.5 ms with the ring.
// The lanes' sums are added through shared memory once per CTA, the CTAs' by the sliced
// reduction, all in a fixed order.
#include "common.cuh"
#include "kernels.h"

namespace bcgs {

namespace {
// Warps that share a row group's sums, row groups of 32 a CTA takes at once, CTAs per SM.
template <int NC>
__host__ __device__ constexpr int pg_parts() { return NC <= 11 ? 1 : (NC <= 16 ? 2 : (NC <= 24 ? 4 : 8)); }
__host__ __device__ constexpr int pg_slots_of(int width) { return width <= 11 ? 4 : (width <= 16 ? 2 : 1); }
template <int NC>
__host__ __device__ constexpr int pg_slots() { return pg_slots_of(NC); }
template <int NC>
__host__ __device__ constexpr int pg_warps() { return pg_parts<NC>() * pg_slots<NC>(); }
__host__ __device__ constexpr int pg_per_sm(int nc) { return nc <= 16 ? 3 : (nc <= 24 ? 2 : 1); }
template <int NC>
__host__ __device__ constexpr int pg_sums() { return NC * (NC + 1) / 2; }
template <int NC>
__host__ __device__ constexpr int pg_ld() { return 32 * pg_slots<NC>() + 1; }
constexpr int PG_ST = 4;   // stages in shared memory of the forms whose registers leave no room for loads ahead
template <int NC>
__host__ __device__ constexpr bool pg_staged() { return pg_slots<NC>() == 1; }
// Part q has columns [pg_cut(q), pg_cut(q + 1)): about as many sums as the others.
template <int NC>
__host__ __device__ constexpr int pg_cut(int q) {
    int j = 0;
    while (j < NC && j * (j + 1) / 2 * pg_parts<NC>() < q * pg_sums<NC>()) ++j;
    return j;
}

// Columns [J0, J1) of the upper Gram over this warp's row groups, into red[sum][lane slot].
template <int NC, int J0, int J1>
__device__ __forceinline__ void panel_sums(const double* __restrict__ V, i64 ld, i64 m, int nc, i64 g0, i64 step,
                                           double* __restrict__ red, int col) {
    constexpr int NA = J1 * (J1 + 1) / 2 - J0 * (J0 + 1) / 2;
    double acc[NA], x[J1];
#pragma unroll
    for (int k = 0; k < NA; ++k) acc[k] = 0.0;
    const i64 groups = (m + 31) / 32;
    auto add = [&] {
        int k = 0;
#pragma unroll
        for (int j = J0; j < J1; ++j)
#pragma unroll
            for (int i = 0; i <= j; ++i, ++k) acc[k] = fma(x[i], x[j], acc[k]);
    };
    if constexpr (pg_staged<NC>()) {
        // red holds PG_ST stages of NC x 32 rows; this warp copies its own columns.
        const int lane = threadIdx.x & 31;
        auto copy = [&](i64 g, int st) {
            const i64 r = g * 32 + lane;
#pragma unroll
            for (int c = J0; c < J1; ++c) {
                const bool ok = c < nc && r < m;
                cp_async8(red + (st * NC + c) * 32 + lane, ok ? V + r + (i64)c * ld : V, ok);
            }
            cp_async_commit();
        };
#pragma unroll
        for (int st = 0; st < PG_ST - 1; ++st) copy(g0 + st * step, st);
        int st = 0;
        for (i64 g = g0; g < groups; g += step) {
            cp_async_wait<PG_ST - 2>();
            // The warps are here at different places of the code: a barrier by its number.
            asm volatile("bar.sync 1, %0;" ::"n"(32 * pg_warps<NC>()) : "memory");
            copy(g + (PG_ST - 1) * step, (st + PG_ST - 1) % PG_ST);
#pragma unroll
            for (int c = 0; c < J1; ++c) x[c] = red[(st * NC + c) * 32 + lane];
            add();
            st = (st + 1) % PG_ST;
        }
        cp_async_wait<0>();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * pg_warps<NC>()) : "memory");
    } else {
        for (i64 g = g0; g < groups; g += step) {
            const i64 r = g * 32 + (threadIdx.x & 31);
#pragma unroll
            for (int c = 0; c < J1; ++c) x[c] = c < nc && r < m ? V[r + (i64)c * ld] : 0.0;
            add();
        }
    }
#pragma unroll
    for (int k = 0; k < NA; ++k) red[(J0 * (J0 + 1) / 2 + k) * pg_ld<NC>() + col] = acc[k];
}

template <int NC, int Q>
__device__ __forceinline__ void panel_part(int part, const double* __restrict__ V, i64 ld, i64 m, int nc, i64 g0,
                                           i64 step, double* __restrict__ red, int col) {
    if (part == Q) {
        panel_sums<NC, pg_cut<NC>(Q), pg_cut<NC>(Q + 1)>(V, ld, m, nc, g0, step, red, col);
        return;
    }
    if constexpr (Q + 1 < pg_parts<NC>()) panel_part<NC, Q + 1>(part, V, ld, m, nc, g0, step, red, col);
}

template <int NC>
__global__ void __launch_bounds__(32 * pg_warps<NC>(), 1)
panel_gram_kernel(const double* __restrict__ V, i64 ld, i64 m, int nc, double* __restrict__ part,
                  const int* __restrict__ gate) {
    extern __shared__ double red[];   // sums x lane slots, then warps x sums
    chain_enter();
    if (gate != nullptr && *gate == 0) return;
    constexpr int SL = pg_slots<NC>(), NS = pg_sums<NC>(), LD = pg_ld<NC>(), NW = pg_warps<NC>();
    constexpr int EACH = 32 * SL / NW;   // lane slots a warp adds
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp % SL;
    // Warps w and w + 4 share an FP64 pipe: of eight parts, pair the ones that add up evenly.
    const int mine = pg_parts<NC>() == 8 ? (0x37650124 >> (4 * warp)) & 7 : warp / SL;
    panel_part<NC, 0>(mine, V, ld, m, nc, (i64)blockIdx.x * SL + slot, (i64)gridDim.x * SL, red, slot * 32 + lane);
    __syncthreads();
    double* sub = red + NS * LD;
    for (int o = lane; o < NS; o += 32) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < EACH; ++k) s += red[o * LD + warp * EACH + k];
        sub[warp * NS + o] = s;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < NS; o += 32 * NW) {
        int j = 0;
        while ((j + 1) * (j + 2) / 2 <= o) ++j;
        const int i = o - j * (j + 1) / 2;
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < NW; w += 4)
            s += (sub[w * NS + o] + sub[(w + 1) * NS + o]) + (sub[(w + 2) * NS + o] + sub[(w + 3) * NS + o]);
        if (j < nc) part[(i64)blockIdx.x * nc * nc + i + (i64)j * nc] = s;
    }
}

// CTAs for nc columns in code of the given width: at least four row groups per warp.
int panel_ctas(i64 m, int nc, int width, int num_sms) {
    const i64 want = ceil_div(ceil_div(m, 32), 4 * pg_slots_of(width)), most = (i64)pg_per_sm(nc) * num_sms;
    return (int)(want < most ? want : most);
}
// Widths there is code for: 8, 10, 12, 14, 16, then every fourth.
constexpr int pg_width(int nc) { return nc <= 8 ? 8 : (nc <= 16 ? (nc + 1) / 2 * 2 : (nc + 3) / 4 * 4); }

template <int NC>
int run_panel(const double* V, i64 ld, i64 m, int nc, double* G, double* part, int num_sms, const int* gate,
              cudaStream_t st) {
    const size_t smem = (size_t)(pg_sums<NC>() * (pg_ld<NC>() + pg_warps<NC>())) * sizeof(double);
    int rc = smem_attr((const void*)panel_gram_kernel<NC>, (int)smem);
    if (rc) return rc;
    const int ctas = panel_ctas(m, nc, NC, num_sms);
    launch_spread(panel_gram_kernel<NC>, (unsigned)ctas, 32 * pg_warps<NC>(), smem, st, V, ld, m, nc, part, gate);
    g_launch_count += 1;
    rc = (int)cudaGetLastError();
    return rc ? rc : launch_gram_reduce_sliced(part, ctas, nc, nc, G, nc, false, st);
}
}  // namespace

i64 panel_gram_part_doubles(i64 m, int s) {
    i64 most = 0;
    for (int nc = 1; nc <= s && nc <= 32; ++nc) {
        const i64 want = (i64)panel_ctas(m, nc, pg_width(nc), kNumSMsDefault) * nc * nc;
        most = want > most ? want : most;
    }
    return most;
}

int launch_panel_gram(const double* X, i64 ld, i64 m, int c0, int nc, double* G, double* part, int num_sms,
                      const int* gate, cudaStream_t st) {
    const double* V = X + (i64)c0 * ld;
    if (num_sms > kNumSMsDefault) num_sms = kNumSMsDefault;   // part's size
    switch (pg_width(nc)) {
#define BCGS_PANEL(N) \
        case N: return run_panel<N>(V, ld, m, nc, G, part, num_sms, gate, st);
        BCGS_PANEL(8) BCGS_PANEL(10) BCGS_PANEL(12) BCGS_PANEL(14) BCGS_PANEL(16) BCGS_PANEL(20) BCGS_PANEL(24)
        BCGS_PANEL(28) BCGS_PANEL(32)
#undef BCGS_PANEL
        default: return (int)cudaErrorInvalidValue;
    }
}

}  // namespace bcgs
