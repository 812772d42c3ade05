// Plain-FP64 tall Gram of the BCGS hot path (the update: update_fp64.cu).
//
// On GB300 the FP64 pipe delivers about 1.2 TFLOP/s (two DFMA per SM per clock),
// while the tall products carry about 16 FLOP per byte of HBM traffic, so the
// product is bound by the FP64 pipe, not by HBM. The kernels are therefore shaped
// for few FP64 instructions, and to reduce deterministically.
//
//   gram_fp64_partial  + gram_reduce : C = X[:, a0:a0+na]^T X[:, b0:b0+nb]
//       replaces the reference's dgemm('T','N') + MPI_Allreduce pair
//       (e.g. SRC/orth.c:182-188). One "synchronization" = one partial pass plus
//       one fixed-order reduction.
#include "batched.h"
#include "common.cuh"
#include "kernels.h"

namespace bcgs {

// ---------------------------------------------------------------------------
// Gram partials. A CTA of 128 threads owns TA columns of A x W = R 128 / TA columns of B
// and walks a contiguous row range of X in stages of GR rows, copied to shared memory
// asynchronously GST stages deep. Thread (ta, tb) keeps R sums: its column of A against
// columns tb, tb + 128 / TA, ... of the W. Partial sums go to part[chunk][i + j * na]
// (column-major na x nb per chunk). Every entry is a sum of FMA chains over the rows of
// the chunk in order, so the result depends on the chunking only, not on TA or R.
//
// One FP64 instruction of a warp occupies its quarter of the SM for 64 clocks, so the
// time is the number of instructions, 4 R per row and CTA, and every column the tile
// has beyond na or nb is paid in full; loads, at most (1 + R) / R per product, are not.
// The tile is therefore chosen per Gram for the least padding (gram_tile below): 32 x 20
// for the 20 columns of blocks of 10, 32 x 4 for blocks of 4, instead of 16 x 32 for all.
// Measured (16 x 32 tiles staged without copies in flight -> now): m = 3001, 64 x 4 97 ->
// 6 us; m = 10^5, 200 x 20 1130 -> 700 us; m = 3 10^5, 272 x 32 4100 -> 3900 us, 1.23 TFLOP/s,
// of which 3 % is the tile below the diagonal.
// ---------------------------------------------------------------------------
namespace {
constexpr int GR = 16;              // X rows per stage
constexpr int GST = 3;              // stages in flight
constexpr int GT_R = 32;            // chunk row ranges are multiples of this
constexpr int GTHREADS = 128;
constexpr int GR_MAX = 8;           // columns of B per thread
constexpr int GSEG = 2048;          // rows of one FMA chain: the chunks of a large m are long, and one
                                    // chain over them would lose digits (one addition per 2048 products)

__host__ __device__ inline int gram_width(int ta, int r) { return r * (GTHREADS / ta); }
__host__ __device__ inline int gram_stage_doubles(int ta, int r) { return GR * ((ta + gram_width(ta, r)) | 1); }
}  // namespace

// The tile at C rows ia0.., C columns jb0.., rows [r_begin, r_end) of X, written to
// `out` (na x nb, ld na). sm holds GST stages of gram_stage_doubles(ta, R).
// Every SEGR rows the running sums are added to a total and restarted, so no FMA
// chain is longer than SEGR rows however long the row range is.
template <int R, int SEGR = GSEG>
__device__ __forceinline__ void gram_partial_body(const double* __restrict__ X, i64 ld, int a0, int na, int b0,
                                                  int nb, int ta, i64 r_begin, i64 r_end, int ia0, int jb0,
                                                  double* __restrict__ out, double* __restrict__ sm) {
    constexpr int SEG = SEGR / GR;  // stages per segment
    static_assert(SEGR > 0 && SEGR % GR == 0, "segments are whole stages");
    const int tbn = GTHREADS / ta, w = R * tbn;
    const int ldr = (ta + w) | 1;
    const int tid = threadIdx.x;
    const int ca = tid & (ta - 1), tb = tid / ta;
    const int nst = r_end > r_begin ? (int)((r_end - r_begin + GR - 1) / GR) : 0;

    // Stage s into its buffer: consecutive threads copy consecutive rows of a column;
    // rows past r_end and columns past na or nb become zeros.
    const int rr = tid % GR, cc0 = tid / GR;
    auto fill = [&](int s) {
        const i64 r = r_begin + (i64)s * GR + rr;
        double* dst = sm + (s % GST) * (GR * ldr) + rr * ldr;
        const bool row = r < r_end;
        for (int cc = cc0; cc < ta + w; cc += GTHREADS / GR) {
            const bool isa = cc < ta;
            const int c = isa ? ia0 + cc : jb0 + cc - ta;
            const bool ok = row && c < (isa ? na : nb);
            cp_async8(dst + cc, ok ? X + r + (i64)((isa ? a0 : b0) + c) * ld : X, ok);
        }
    };
    double acc[R], tot[R];
#pragma unroll
    for (int k = 0; k < R; ++k) { acc[k] = 0.0; tot[k] = 0.0; }
#pragma unroll
    for (int s = 0; s < GST - 1; ++s) {
        if (s < nst) fill(s);
        cp_async_commit();
    }
    // (Segments are an outer loop: additions behind a condition in the stage loop would
    // be predicated off, and still take their 64 clocks, at every stage.)
    for (int s0 = 0; s0 < nst; s0 += SEG) {
        const int s1 = min(nst, s0 + SEG);
#pragma unroll 1
        for (int s = s0; s < s1; ++s) {
            cp_async_wait<GST - 2>();
            __syncthreads();   // stage s is here, and every thread is done with stage s - 1
            if (s + GST - 1 < nst) fill(s + GST - 1);
            cp_async_commit();
            const double* pa = sm + (s % GST) * (GR * ldr) + ca;
            const double* pb = pa - ca + ta + tb;
#pragma unroll 4
            for (int q = 0; q < GR; ++q) {
                const double av = pa[q * ldr];
#pragma unroll
                for (int k = 0; k < R; ++k) acc[k] = fma(av, pb[q * ldr + k * tbn], acc[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k) { tot[k] += acc[k]; acc[k] = 0.0; }
    }
    const int i = ia0 + ca;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int j = jb0 + tb + k * tbn;
        if (i < na && j < nb) out[i + (i64)j * na] = tot[k];
    }
}

// Tile (ta, r) of a Gram and the number of its tiles that are not skipped. With
// `upper` (>= 0: b0 - a0) only entries on or above the diagonal of X^T X are needed, and
// tiles wholly below it are left out (their part is not written).
struct GramTile {
    int ta = 32, r = 1, tilesA = 1, tilesB = 1;
    i64 live = 1;
};
// Strips of A a tile column (columns [jb w, (jb + 1) w) of the nb) has above the diagonal.
__host__ __device__ inline int gram_live_strips(int upper, int jb, int w, int nb, int ta, int tilesA) {
    if (upper < 0) return tilesA;
    const int end = upper + (jb * w + w < nb ? jb * w + w : nb);
    const int hi = (end + ta - 1) / ta;
    return hi < tilesA ? hi : tilesA;
}
// Live tile t: its strip and column, counted column by column.
__device__ __forceinline__ void gram_tile_of(int t, int upper, int w, int nb, int ta, int tilesA, int& ia0, int& jb0) {
    int jb = 0;
    for (;; ++jb) {
        const int hi = gram_live_strips(upper, jb, w, nb, ta, tilesA);
        if (t < hi) break;
        t -= hi;
    }
    ia0 = t * ta;
    jb0 = jb * w;
}
static GramTile gram_tile(int na, int nb, int upper) {
    GramTile best;
    i64 best_cost = -1, best_loads = 0;
    for (int ta = 16; ta <= 64; ta *= 2)
        for (int r = 1; r <= GR_MAX; ++r) {
            const int w = gram_width(ta, r);
            if (r > 1 && gram_width(ta, r - 1) >= nb) break;
            GramTile t;
            t.ta = ta; t.r = r;
            t.tilesA = (int)ceil_div(na, ta); t.tilesB = (int)ceil_div(nb, w);
            t.live = 0;
            for (int jb = 0; jb < t.tilesB; ++jb) t.live += gram_live_strips(upper, jb, w, nb, ta, t.tilesA);
            const i64 cost = t.live * r, loads = t.live * (ta + w);
            if (best_cost < 0 || cost < best_cost || (cost == best_cost && loads < best_loads)) {
                best_cost = cost; best_loads = loads;
                best = t;
            }
        }
    return best;
}

// blockIdx: chunk, live tile (no CTA for a skipped one: an SM that got one would be left
// with less than its share while others take one more). A wide C has more than 65535
// tiles, which go on in z.
template <int R, int SEGR>
__global__ void __launch_bounds__(GTHREADS)
gram_fp64_partial(const double* __restrict__ X, i64 ld, i64 m, int a0, int na, int b0, int nb, int ta, int upper,
                  int live, i64 rows_per_chunk, double* __restrict__ part, const int* __restrict__ gate) {
    extern __shared__ double sm[];
    chain_enter();
    if (gate != nullptr && *gate == 0) return;
    const int chunk = blockIdx.x;
    const int t = (int)(blockIdx.y + blockIdx.z * gridDim.y);
    if (t >= live) return;
    int ia0, jb0;
    gram_tile_of(t, upper, gram_width(ta, R), nb, ta, (na + ta - 1) / ta, ia0, jb0);
    const i64 r_begin = (i64)chunk * rows_per_chunk;
    const i64 r_end = min(m, r_begin + rows_per_chunk);
    gram_partial_body<R, SEGR>(X, ld, a0, na, b0, nb, ta, r_begin, r_end, ia0, jb0, part + (i64)chunk * na * nb, sm);
}

template <int SEGR>
static int launch_partial(const GramTile& t, int nchunks, const double* X, i64 ld, i64 m, int a0, int na, int b0,
                          int nb, int upper, i64 rows, double* part, const int* gate, cudaStream_t st) {
    const i64 layers = ceil_div(t.live, 65535);
    const dim3 grid((unsigned)nchunks, (unsigned)ceil_div(t.live, layers), (unsigned)layers);
    const size_t smem = (size_t)GST * gram_stage_doubles(t.ta, t.r) * sizeof(double);
    switch (t.r) {
#define BCGS_GP(RR)                                                                                               \
    case RR:                                                                                                      \
        launch_spread(gram_fp64_partial<RR, SEGR>, grid, GTHREADS, smem, st, X, ld, m, a0, na, b0, nb, t.ta, upper, \
                      (int)t.live, rows, part, gate);                                                             \
        break;
        BCGS_GP(1) BCGS_GP(2) BCGS_GP(3) BCGS_GP(4) BCGS_GP(5) BCGS_GP(6) BCGS_GP(7) BCGS_GP(8)
#undef BCGS_GP
        default: return (int)cudaErrorInvalidValue;
    }
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

// Fixed-order sum over chunks: out[i + j*ldo] = sum_{c=0}^{nchunks-1} part[c][i + j*na].
// Each entry is summed sequentially in chunk order, so results are bit-identical
// run to run for a given (m, na, nb). The chain of additions is short next to the
// latency of the loads that feed it, so RD_AHEAD loads are issued ahead of the
// additions, and the CTAs are small so that a few thousand entries reach most SMs.
// m = 10^5, na x nb = 200 x 20, about 190 chunks: 25 us (33 us with the loads issued
// four at a time from 256-thread CTAs).
constexpr int RD_THREADS = 64;
constexpr int RD_AHEAD = 16;

__device__ __forceinline__ void gram_reduce_body(const double* __restrict__ part, int nchunks, int na, int nb,
                                                 double* __restrict__ out, int ldo, i64 blk) {
    const i64 total = (i64)na * nb;
    const i64 e = blk * RD_THREADS + threadIdx.x;
    if (e >= total) return;
    const double* p = part + e;
    double s = 0.0, v[RD_AHEAD], n[RD_AHEAD];
    int c = 0;
    if (nchunks >= RD_AHEAD) {
#pragma unroll
        for (int k = 0; k < RD_AHEAD; ++k) v[k] = p[(i64)k * total];
        for (; c + 2 * RD_AHEAD <= nchunks; c += RD_AHEAD) {
#pragma unroll
            for (int k = 0; k < RD_AHEAD; ++k) n[k] = p[(i64)(c + RD_AHEAD + k) * total];
#pragma unroll
            for (int k = 0; k < RD_AHEAD; ++k) s += v[k];
#pragma unroll
            for (int k = 0; k < RD_AHEAD; ++k) v[k] = n[k];
        }
#pragma unroll
        for (int k = 0; k < RD_AHEAD; ++k) s += v[k];
        c += RD_AHEAD;
    }
#pragma unroll
    for (int k = 0; k < RD_AHEAD; ++k) v[k] = c + k < nchunks ? p[(i64)(c + k) * total] : 0.0;
#pragma unroll 1
    for (int k = 0; c < nchunks; ++c, ++k) {
        double x = v[0];
#pragma unroll
        for (int q = 1; q < RD_AHEAD; ++q)
            if (q == k) x = v[q];
        s += x;
    }
    out[e % na + (e / na) * ldo] = s;
}

__global__ void __launch_bounds__(RD_THREADS)
gram_reduce(const double* __restrict__ part, int nchunks, int na, int nb, double* __restrict__ out, int ldo) {
    chain_enter();
    gram_reduce_body(part, nchunks, na, nb, out, ldo, blockIdx.x);
}

// The same sum by RS_SLICES threads per entry, each over a contiguous range of chunks, the
// ranges then added in order: a shorter chain for the reductions whose order nothing
// ties to a sequential one (the split forms' partials, exact up to here, and the
// narrow panels' Grams). 150 chunks of 100 x 20: 7 -> 3.5 us.
constexpr int RS_SLICES = 8;
constexpr int RS_OUTS = 32;

__device__ __forceinline__ void gram_reduce_sliced_body(const double* __restrict__ part, int nchunks, int na, int nb,
                                                        double* __restrict__ out, int ldo, i64 blk) {
    __shared__ double red[RS_SLICES][RS_OUTS];
    const i64 total = (i64)na * nb;
    const int lane = threadIdx.x % RS_OUTS, slice = threadIdx.x / RS_OUTS;
    const i64 e = blk * RS_OUTS + lane;
    double s = 0.0;
    if (e < total) {
        const int per = (nchunks + RS_SLICES - 1) / RS_SLICES;
        const int c1 = min(nchunks, (slice + 1) * per);
        int c = slice * per;
        for (; c + 8 <= c1; c += 8) {
            double v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = part[(i64)(c + k) * total + e];
#pragma unroll
            for (int k = 0; k < 8; ++k) s += v[k];
        }
#pragma unroll 1
        for (; c < c1; ++c) s += part[(i64)c * total + e];
    }
    red[slice][lane] = s;
    __syncthreads();
    if (slice != 0 || e >= total) return;
#pragma unroll
    for (int k = 1; k < RS_SLICES; ++k) s += red[k][lane];
    out[e % na + (e / na) * ldo] = s;
}

__global__ void __launch_bounds__(RS_SLICES * RS_OUTS)
gram_reduce_sliced(const double* __restrict__ part, int nchunks, int na, int nb, double* __restrict__ out, int ldo) {
    chain_enter();
    gram_reduce_sliced_body(part, nchunks, na, nb, out, ldo, blockIdx.x);
}

int gram_reduce_sliced_ctas(int na, int nb) { return (int)ceil_div((i64)na * nb, RS_OUTS); }

int launch_gram_reduce_sliced(const double* part, int nchunks, int na, int nb, double* out, int ldo, bool counted,
                              cudaStream_t st) {
    launch_chained(gram_reduce_sliced, (unsigned)gram_reduce_sliced_ctas(na, nb), RS_SLICES * RS_OUTS, 0, st, part,
                   nchunks, na, nb, out, ldo);
    g_launch_count += 1;
    if (counted) g_reduce_count += 1;
    return (int)cudaGetLastError();
}

int gram_reduce_ctas(int na, int nb) { return (int)ceil_div((i64)na * nb, RD_THREADS); }

// Rows per Gram chunk forced by orth_gb300_set_gram_chunk_rows (0: the default
// policy below).
long long g_gram_chunk_rows = 0;

// Doubles of partials a Gram may take: at most what a full SM's worth of 16 x 32 tiles
// per SM would (for narrower B in proportion), and chunks of no fewer than GC_MIN rows.
constexpr int GC_MIN = 64;
static i64 gram_part_cap(int nb) { return 16LL * kNumSMsDefault * 16 * (nb < 32 ? nb : 32); }

i64 gram_part_doubles_fp64(i64 m, int na_max, int nb_max) {
    const i64 one = (i64)na_max * nb_max;
    if (g_gram_chunk_rows > 0) return ceil_div(m, g_gram_chunk_rows) * one + 1024;
    const i64 cap = gram_part_cap(nb_max), all = ceil_div(m, GC_MIN) * one;
    const i64 most = cap < all ? cap : all;
    return (most > one ? most : one) + 1024;
}

// Chunks: the CTAs (live tiles x chunks, equal work each) are laid on the SMs in w
// rounds, w = 1 .. 16, as many as fit; a round of L rows takes 64 R L clocks on each
// SM quarter, and every chunk adds about 130 clocks to the reduction's chain. More
// rounds mean fewer SMs idle in the last one and shorter chains, fewer mean fewer
// partials. One CTA of four warps keeps the FP64 pipe 63 % busy (its barriers and loads
// have nothing beside them), two 91 %, three 97 % (ncu, m = 10^5, na x nb = 100 x 10 to
// 200 x 8).
static int gram_chunks(i64 m, int na, int nb, const GramTile& t, int num_sms) {
    if (g_gram_chunk_rows > 0) {
        const i64 c = ceil_div(m, g_gram_chunk_rows);
        return (int)(c < 1 ? 1 : c);
    }
    const i64 one = (i64)na * nb;
    i64 cmax = gram_part_cap(nb) / one;
    const i64 crows = ceil_div(m, GC_MIN);
    if (cmax > crows) cmax = crows;
    if (cmax > 4096) cmax = 4096;
    if (cmax < 1) cmax = 1;
    i64 best = 1;
    double best_cost = 0.0;
    for (int w = 1; w <= 16; ++w) {
        i64 c = (i64)w * num_sms / t.live;
        if (c < 1) c = 1;
        if (c > cmax) c = cmax;
        const i64 rows = ceil_div(ceil_div(m, c), GT_R) * GT_R;
        c = ceil_div(m, rows);
        const double rounds = (double)ceil_div(c * t.live, num_sms);
        const double busy = rounds < 1.5 ? 0.63 : (rounds < 2.5 ? 0.91 : 0.97);
        const double cost = rounds * (64.0 * t.r * (double)rows / busy + 1000.0) + 130.0 * (double)c;
        if (w == 1 || cost < best_cost) { best = c; best_cost = cost; }
    }
    return (int)best;
}

int launch_gram_fp64(const double* X, i64 ld, i64 m, int a0, int na, int b0, int nb, double* out, int ldo,
                     double* part, bool upper_only, int num_sms, cudaStream_t st, const int* gate, bool counted) {
    if (na <= 0 || nb <= 0) return 0;
    const int upper = upper_only ? b0 - a0 : -1;
    const GramTile t = gram_tile(na, nb, upper);
    const int nchunks = gram_chunks(m, na, nb, t, num_sms);
    i64 rows_per_chunk = ceil_div(m, nchunks);
    rows_per_chunk = ceil_div(rows_per_chunk, GT_R) * GT_R;
    const int rc = launch_partial<GSEG>(t, nchunks, X, ld, m, a0, na, b0, nb, upper, rows_per_chunk, part, gate,
                                   st);
    if (rc) return rc;
    if (!counted) g_reduce_count -= 1;   // launch_gram_reduce counts it
    return launch_gram_reduce(part, nchunks, na, nb, out, ldo, st);
}

int launch_gram_partials_fp64(const double* X, i64 ld, i64 m, int a0, int na, int b0, int nb, double* part,
                              i64 rows, cudaStream_t st) {
    if (na <= 0 || nb <= 0 || m <= 0) return 0;
    if (rows <= 0 || rows % GT_R != 0) return (int)cudaErrorInvalidValue;
    return launch_partial<256>(gram_tile(na, nb, -1), (int)ceil_div(m, rows), X, ld, m, a0, na, b0, nb, -1, rows, part,
                               nullptr, st);
}

int launch_gram_reduce(const double* part, int nchunks, int na, int nb, double* out, int ldo,
                       cudaStream_t st) {
    launch_chained(gram_reduce, (unsigned)gram_reduce_ctas(na, nb), RD_THREADS, 0, st, part, nchunks, na, nb, out, ldo);
    g_launch_count += 1;
    g_reduce_count += 1;
    return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Batched forms: one launch over many matrices' jobs (batched.h).
// ---------------------------------------------------------------------------
int gram_batched_tile(int na, int b0, int nb, int* ta, int* r) {
    const GramTile t = gram_tile(na, nb, b0);
    *ta = t.ta; *r = t.r;
    return (int)t.live;
}

// Job j's CTAs: chunk fastest, then live tile.
__global__ void __launch_bounds__(GTHREADS)
gram_partial_batched(const GramJob* __restrict__ jobs, const int* __restrict__ prefix, int njobs) {
    extern __shared__ double sm[];
    const int j = batched_job_of(prefix, njobs, blockIdx.x);
    const GramJob J = jobs[j];
    const int local = blockIdx.x - prefix[j];
    const int chunk = local % J.nchunks;
    const int t = local / J.nchunks;
    int ia0, jb0;
    gram_tile_of(t, J.b0, gram_width(J.ta, J.r), J.nb, J.ta, (J.na + J.ta - 1) / J.ta, ia0, jb0);
    const i64 r_begin = (i64)chunk * J.rows_per_chunk;
    const i64 r_end = min(J.m, r_begin + J.rows_per_chunk);
    double* out = J.part + (i64)chunk * J.na * J.nb;
    switch (J.r) {
#define BCGS_GB(RR) \
    case RR: gram_partial_body<RR>(J.X, J.ld, 0, J.na, J.b0, J.nb, J.ta, r_begin, r_end, ia0, jb0, out, sm); break;
        BCGS_GB(1) BCGS_GB(2) BCGS_GB(3) BCGS_GB(4) BCGS_GB(5) BCGS_GB(6) BCGS_GB(7) BCGS_GB(8)
#undef BCGS_GB
    }
}

// Each job's sum in the single launch's order (items: gram_reduce_ctas per job).
__global__ void __launch_bounds__(RD_THREADS)
gram_reduce_batched(const GramJob* __restrict__ jobs, const int* __restrict__ prefix, int njobs) {
    const int j = batched_job_of(prefix, njobs, blockIdx.x);
    const GramJob& J = jobs[j];
    gram_reduce_body(J.part, J.nchunks, J.na, J.nb, J.C, J.ldc, blockIdx.x - prefix[j]);
}

__global__ void __launch_bounds__(RS_SLICES * RS_OUTS)
gram_reduce_sliced_batched(const GramJob* __restrict__ jobs, const int* __restrict__ prefix, int njobs) {
    const int j = batched_job_of(prefix, njobs, blockIdx.x);
    const GramJob& J = jobs[j];
    gram_reduce_sliced_body(J.part, J.nchunks, J.na, J.nb, J.C, J.ldc, blockIdx.x - prefix[j]);
}

int launch_gram_reduce_sliced_batched(const GramJob* jobs, const int* prefix, int njobs, int items, cudaStream_t st) {
    if (items <= 0) return 0;
    gram_reduce_sliced_batched<<<(unsigned)items, RS_SLICES * RS_OUTS, 0, st>>>(jobs, prefix, njobs);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

int launch_gram_partial_batched(const GramJob* jobs, const int* prefix, int njobs, int items, cudaStream_t st) {
    if (items <= 0) return 0;
    // Stages for the widest tile a batch's blocks (s <= 16) can take.
    constexpr size_t smem = (size_t)GST * GR * ((64 + 2 * GR_MAX) | 1) * sizeof(double);
    gram_partial_batched<<<(unsigned)items, GTHREADS, smem, st>>>(jobs, prefix, njobs);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

int launch_gram_reduce_batched(const GramJob* jobs, const int* prefix, int njobs, int items, cudaStream_t st) {
    if (items <= 0) return 0;
    gram_reduce_batched<<<(unsigned)items, RD_THREADS, 0, st>>>(jobs, prefix, njobs);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

}  // namespace bcgs
