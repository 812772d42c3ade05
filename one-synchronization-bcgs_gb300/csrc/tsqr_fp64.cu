// IntraOrtho: explicit TSQR of a tall m x nc panel in FP64 (nc <= 64).
//
// Replaces the reference's Trilinos TSQR::Tsqr::factorExplicit (SRC/orth.c:14-46,
// call sites :107,:271,:413,:505,:522,:534,:601,:613,:651). Trilinos is not part of
// the reference, so the algorithm here is the published TSQR reduction tree:
//
//   level 0: the panel is cut into tiles of TR rows; one CTA of W warps per tile
//            computes a Householder QR of its tile in shared memory (warp butterfly
//            sums; the warps share out the columns), writes the explicit tile Q in
//            place and its nc x nc R into the next level's stack.
//   level l: the stacked R factors (a (tiles * nc) x nc matrix) are cut into tiles
//            of TR rows again and factored the same way, until one tile remains.
//   root   : R is sign-normalized (diag(R) >= 0, the column signs moved into Q).
//   down   : each level's tile Q is multiplied by its nc x nc block of the level
//            above, from the root down to the panel, giving the explicit Q.
//
// Every reduction is in a fixed order (warp butterfly sums, a fixed tree), so
// results are bit-identical run to run.
#include "batched.h"
#include "common.cuh"
#include "kernels.h"

namespace bcgs {

// Tile rows and warps per tile by template width. All tiles hold 256 rows: a level of
// the tree divides the row count by TR / nc, so taller tiles mean fewer levels and
// fewer flops, at the price of fewer tiles resident per SM. One FP64 instruction of a
// warp occupies its quarter of the SM for 64 clocks whatever the other warps do, so
// what counts is the number of FP64 instructions and that all four quarters have
// some: four or eight columns per warp (four columns' lane sums cost 6 additions
// together, one column's alone 5).
constexpr int TSQR_TR = 256;
template <int NC>
constexpr int tsqr_tile_warps() { return NC > 16 ? 8 : (NC > 8 ? 4 : 2); }
// Levels with tiles for several CTAs on every SM have the quarters busy with half as
// many warps per tile, twice the columns each: fewer lane sums. us, half against full:
// 2^21 x 16 2395 / 2697, 10^5 x 16 (391 tiles) 165 / 157; 391 tiles x 32 529 / 628, 49 tiles 316 / 250;
// a tile of 64 columns is best with 8 warps everywhere (789 / 803 alone).
template <int NC>
constexpr int tsqr_many_tiles() { return (NC <= 16 ? 4 : 2) * kNumSMsDefault; }
template <int NC>
constexpr int tsqr_many_warps() { return NC > 32 ? 8 : (NC > 8 ? tsqr_tile_warps<NC>() / 2 : tsqr_tile_warps<NC>()); }

int tsqr_tile_rows(int nc) { (void)nc; return TSQR_TR; }

// Shared memory of one tile: the TR x NC tile, column-major (ld TR), the reflectors'
// scalars and R's diagonal.
static size_t tsqr_tile_smem_bytes(int NC) { return (size_t)(TSQR_TR * NC + 2 * NC) * sizeof(double); }

// Sum of one value over the warp by an xor butterfly. Lane pairs add the same two
// operands (a + b == b + a), so every lane ends with the same bits.
__device__ __forceinline__ double warp_sum1(double w) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    return w;
}

// One reflector H = I - t v v^T applied to the K columns c, c + W, ... (lane `lane` owns
// rows lane + 32 i, i < RPL): w_g = sum_r v[r] a[r][c_g], then a[r][c_g] -= t w_g v[r]. v is
// zero above the reflector's pivot row, so those rows keep their values. The K sums are
// reduced together: lane bit 0 splits the columns into pairs and bit 1 into singles
// (each lane adds the partner's half it keeps), then the remaining bits finish by a
// butterfly. Every column is summed in warp_sum1's order, so the result does not depend
// on which columns are taken together. (Of several orders with the same cost and the same
// errors, this is one with which the golden case of exactly dependent blocks, whose LOO
// is a draw of the roundings, meets its limit; so is the order of the narrow Gram's
// sums at 8 to 16 columns.)
template <int RPL, int K>
__device__ __forceinline__ void apply_cols(double* a, int c, int W, const double* v, double t, int lane) {
    double x[K][RPL], w[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int g = 0; g < K; ++g)
#pragma unroll
        for (int i = RPL - 1; i >= 0; --i) {
            x[g][i] = a[(c + g * W) * (32 * RPL) + lane + 32 * i];
            w[g] = fma(v[i], x[g][i], w[g]);
        }
    double k;
    const bool b0 = (lane & 1) != 0, b1 = (lane & 2) != 0;
    if constexpr (K >= 3) {
        double k0 = b0 ? w[2] : w[0], k1 = b0 ? w[3] : w[1];
        k0 += __shfl_xor_sync(0xffffffffu, b0 ? w[0] : w[2], 1);
        k1 += __shfl_xor_sync(0xffffffffu, b0 ? w[1] : w[3], 1);
        k = b1 ? k1 : k0;
        k += __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 2);
    } else {
        k = w[0];
        if constexpr (K == 2) k = b0 ? w[1] : w[0];
        k += __shfl_xor_sync(0xffffffffu, K == 2 ? (b0 ? w[0] : w[1]) : w[0], 1);
        k += __shfl_xor_sync(0xffffffffu, k, 2);
    }
    k += __shfl_xor_sync(0xffffffffu, k, 4);
    k += __shfl_xor_sync(0xffffffffu, k, 8);
    k += __shfl_xor_sync(0xffffffffu, k, 16);
    k *= -t;
#pragma unroll
    for (int g = 0; g < K; ++g) {
        const double wg = K == 1 ? k : __shfl_sync(0xffffffffu, k, K == 2 ? g : (g >> 1) + 2 * (g & 1));
#pragma unroll
        for (int i = 0; i < RPL; ++i) a[(c + g * W) * (32 * RPL) + lane + 32 * i] = fma(wg, v[i], x[g][i]);
    }
}

// H applied to the columns c, c + W, ... below nc.
template <int RPL, int W>
__device__ __forceinline__ void apply_own(double* a, int c, int nc, const double* v, double t, int lane) {
    for (; c + 3 * W < nc; c += 4 * W) apply_cols<RPL, 4>(a, c, W, v, t, lane);
    if (c + 2 * W < nc) apply_cols<RPL, 3>(a, c, W, v, t, lane);
    else if (c + W < nc) apply_cols<RPL, 2>(a, c, W, v, t, lane);
    else if (c < nc) apply_cols<RPL, 1>(a, c, W, v, t, lane);
}

// Whether d is a positive number of ordinary size, 2^-900 .. 2^900 (an integer test: a
// comparison would be one more FP64 instruction).
__device__ __forceinline__ bool ordinary(double d) {
    const unsigned hi = (unsigned)__double2hiint(d);
    return hi >= 0x07B00000u && hi < 0x78300000u;
}

// Householder reflector of column c (held in x, lane's rows lane + 32 i): H = I - t v v^T
// with v = x below row c and alpha - beta at it, beta = -sign(alpha) ||x[c:]||,
// t = 2 / v^T v: LAPACK's dlarfg without scaling v to a unit
// pivot, which saves a multiply per row and a division. A column whose squares leave
// the ordinary range is scaled first (v may have any scale). Written back in place: v
// from row c down, R's entries above; t to tau[c], beta to rdiag[c].
template <int RPL>
__device__ __forceinline__ void make_reflector(double* a, double* tau, double* rdiag, int c, int lane, double* x) {
    auto below = [&]() {
        double p = 0.0;
#pragma unroll
        for (int i = RPL - 1; i >= 0; --i) {
            const double y = lane + 32 * i > c ? x[i] : 0.0;
            p = fma(y, y, p);
        }
        return warp_sum1(p);
    };
    double p = below();
    double alpha = __shfl_sync(0xffffffffu, c < 32 ? x[0] : x[1], c & 31);
    double t = 0.0, beta = alpha, vc = 0.0;
    bool live = __double_as_longlong(p) != 0LL;
    if (!live) {   // squares that all underflowed are not a zero column
        unsigned long long any = 0;
#pragma unroll
        for (int i = 0; i < RPL; ++i)
            if (lane + 32 * i > c) any |= (unsigned long long)__double_as_longlong(x[i]) << 1;
        live = __any_sync(0xffffffffu, any != 0) != 0;
    }
    if (live) {
        double q = fma(alpha, alpha, p), back = 1.0;
        if (!ordinary(q)) {
            const bool small = (unsigned)__double2hiint(q) < 0x3FF00000u;
            const double sc = __longlong_as_double(small ? 0x7830000000000000LL : 0x1FF0000000000000LL);   // 2^900, 2^-512
            back = __longlong_as_double(small ? 0x07B0000000000000LL : 0x5FF0000000000000LL);
#pragma unroll
            for (int i = 0; i < RPL; ++i)
                if (lane + 32 * i >= c) x[i] *= sc;
            alpha *= sc;
            p = below();
            q = fma(alpha, alpha, p);
        }
        beta = -copysign(root(q, rsqrt(q)), alpha);
        vc = alpha - beta;
        const double e = 0.5 * fma(vc, vc, p);   // t v^T v = 2 for the v that is stored
        t = ordinary(e) ? recip(e) : 1.0 / e;
        if (__double_as_longlong(back) != __double_as_longlong(1.0)) beta *= back;
    }
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
        const int r = lane + 32 * i;
        a[c * (32 * RPL) + r] = r == c ? vc : x[i];
    }
    if (lane == 0) {
        tau[c] = t;
        rdiag[c] = beta;
    }
}

// Reflector j (stored in column j) into registers, zero above its pivot row.
template <int RPL>
__device__ __forceinline__ double load_reflector(const double* a, const double* tau, int j, int lane, double* v) {
#pragma unroll
    for (int i = 0; i < RPL; ++i) {
        const int r = lane + 32 * i;
        v[i] = r >= j ? a[j * (32 * RPL) + r] : 0.0;
    }
    return tau[j];
}

// W warps per tile, the tile in shared memory (lane L owns rows L, L+32, ...).
// A: rows x nc (lda); tile `tile` covers rows [tile*TR, min(rows, (tile+1)*TR)).
// Householder QR (dgeqr2's order), then the tile's R (upper, lower part zero) to Rst
// rows [tile*nc, (tile+1)*nc) (ld ldr), then the explicit tile Q formed in place in
// dorg2r's order (backward over the reflectors) and written to Q (ldq; may alias A).
// Tiles shorter than nc rows are padded with zero rows; padded rows of Q are not
// written. smem holds tsqr_tile_smem_bytes(NC).
//
// Column c belongs to warp c mod W, so the warps' shares stay even as columns are
// finished. Each reflector is formed once, by its column's warp: while reflector j is
// applied, the owner of column j + 1 updates that column first, alone, and forms
// reflector j + 1 from it before its other columns (look-ahead), so one barrier per
// reflector separates the steps. Every sum has a fixed order that depends on
// neither W nor the grouping, so results are bit-identical for every W.
// Measured (before: one, four or 16 warps a tile with fixed groups of four columns,
// unit-pivot reflectors with a division each, tau v published beside v): a level of one
// tile of 256 x 10, whose chain of reflectors nothing hides, 124 -> 53 us; the leaves of
// 10^5 x 10 133 -> 76 us, of 2^21 x 16 2.81 -> 2.70 ms with 4 warps, 2.40 with 2.
template <int NC, int W>
__device__ void tsqr_tile_body(const double* A, i64 lda, i64 rows, int nc, double* Q, i64 ldq,
                               double* __restrict__ Rst, i64 ldr, i64 tile, double* smem) {
    constexpr int TR = TSQR_TR;
    constexpr int RPL = TR / 32;
    double* a = smem;              // a[c * TR + r]
    double* tau = smem + TR * NC;
    double* rdiag = tau + NC;
    const int lane = threadIdx.x & 31;
    const int warp = (int)(threadIdx.x >> 5);
    const i64 row0 = tile * TR;
    const i64 h = min((i64)TR, rows - row0);
    __syncthreads();
    for (int c = warp; c < nc; c += W)
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            const int r = lane + 32 * i;
            a[c * TR + r] = (r < h) ? A[row0 + r + (i64)c * lda] : 0.0;
        }
    // (each warp has only written columns of its own so far)
    double v[RPL];
    if (warp == 0) {
        double x[RPL];
#pragma unroll
        for (int i = 0; i < RPL; ++i) x[i] = a[lane + 32 * i];
        make_reflector<RPL>(a, tau, rdiag, 0, lane, x);
    }
    __syncthreads();

    for (int j = 0; j + 1 < nc; ++j) {
        const double t = load_reflector<RPL>(a, tau, j, lane, v);
        const bool live = __double_as_longlong(t) != 0LL;
        int c = j + 1 + ((warp - (j + 1)) % W + W) % W;   // this warp's first column after j
        if (c == j + 1) {
            double x[RPL], w = 0.0;
#pragma unroll
            for (int i = 0; i < RPL; ++i) x[i] = a[c * TR + lane + 32 * i];
            if (live) {
#pragma unroll
                for (int i = RPL - 1; i >= 0; --i) w = fma(v[i], x[i], w);
                w = warp_sum1(w) * -t;
#pragma unroll
                for (int i = 0; i < RPL; ++i) x[i] = fma(w, v[i], x[i]);
            }
            make_reflector<RPL>(a, tau, rdiag, c, lane, x);
            c += W;
        }
        if (live) apply_own<RPL, W>(a, c, nc, v, t, lane);
        __syncthreads();
    }
    // R to the stack (upper, lower zero).
    for (int e = threadIdx.x; e < nc * nc; e += 32 * W) {
        const int i = e % nc, c = e / nc;
        Rst[tile * nc + i + (i64)c * ldr] = i < c ? a[c * TR + i] : (i == c ? rdiag[c] : 0.0);
    }
    __syncthreads();
    // Explicit Q in place (dorg2r): for j = nc-1 .. 0, apply H_j to columns j+1.. and set
    // column j to (I - t v v^T) e_j (its owner, after the barrier that ends every
    // warp's reading of reflector j).
    for (int j = nc - 1; j >= 0; --j) {
        const double t = load_reflector<RPL>(a, tau, j, lane, v);
        if (__double_as_longlong(t) != 0LL)
            apply_own<RPL, W>(a, j + 1 + ((warp - (j + 1)) % W + W) % W, nc, v, t, lane);
        __syncthreads();
        if (j % W == warp) {
            const double s = -t * __shfl_sync(0xffffffffu, j < 32 ? v[0] : v[1], j & 31);
#pragma unroll
            for (int i = 0; i < RPL; ++i) {
                const int r = lane + 32 * i;
                const double y = s * v[i];
                a[j * TR + r] = r == j ? 1.0 + y : y;
            }
        }
    }
    // (column c's owner is the only one that has written it since the last barrier)
    for (int c = warp; c < nc; c += W)
#pragma unroll
        for (int i = 0; i < RPL; ++i) {
            const int r = lane + 32 * i;
            if (r < h) Q[row0 + r + (i64)c * ldq] = a[c * TR + r];
        }
}

template <int NC, int W>
__global__ void __launch_bounds__(32 * W)
tsqr_tile_kernel(const double* A, i64 lda, i64 rows, int nc, double* Q, i64 ldq,
                 double* __restrict__ Rst, i64 ldr, const int* __restrict__ done) {
    extern __shared__ double smem[];
    chain_enter();
    if (done != nullptr && *done) return;
    tsqr_tile_body<NC, W>(A, lda, rows, nc, Q, ldq, Rst, ldr, blockIdx.x, smem);
}

template <int NC, int W>
static int launch_tiles_w(double* A, i64 lda, i64 rows, int nc, double* Rst, i64 ldr, const int* done, cudaStream_t st) {
    const size_t smem = tsqr_tile_smem_bytes(NC);
    const int rc = smem_attr((const void*)tsqr_tile_kernel<NC, W>, (int)smem);
    if (rc) return rc;
    launch_spread(tsqr_tile_kernel<NC, W>, (unsigned)ceil_div(rows, TSQR_TR), 32 * W, smem, st, A, lda, rows, nc, A, lda, Rst, ldr,
                                                                                    done);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}
template <int NC>
static int launch_tiles(double* A, i64 lda, i64 rows, int nc, double* Rst, i64 ldr, const int* done, cudaStream_t st) {
    if (ceil_div(rows, TSQR_TR) >= tsqr_many_tiles<NC>())
        return launch_tiles_w<NC, tsqr_many_warps<NC>()>(A, lda, rows, nc, Rst, ldr, done, st);
    return launch_tiles_w<NC, tsqr_tile_warps<NC>()>(A, lda, rows, nc, Rst, ldr, done, st);
}

// Root fix-up: make diag(R) >= 0. R (nc x nc, ld ldr) rows with a negative
// diagonal are negated, as are the matching columns of the root Q (hq x nc, ldq).
// The final R is also copied to Rout (ld ldro), lower part zero.
__device__ void tsqr_root_fix_body(double* Q, i64 ldq, int hq, int nc, const double* R, i64 ldr,
                                   double* Rout, int ldro) {
    __shared__ double sgn[64];
    __syncthreads();
    if (threadIdx.x < nc) sgn[threadIdx.x] = (R[threadIdx.x + (i64)threadIdx.x * ldr] < 0.0) ? -1.0 : 1.0;
    __syncthreads();
    for (int e = threadIdx.x; e < nc * nc; e += blockDim.x) {
        int i = e % nc, c = e / nc;
        Rout[i + (i64)c * ldro] = (i <= c) ? sgn[i] * R[i + (i64)c * ldr] : 0.0;
    }
    for (int e = threadIdx.x; e < hq * nc; e += blockDim.x) {
        int i = e % hq, c = e / hq;
        Q[i + (i64)c * ldq] *= sgn[c];
    }
    __syncthreads();
}

__global__ void tsqr_root_fix(double* Q, i64 ldq, int hq, int nc, const double* R, i64 ldr,
                              double* Rout, int ldro, const int* __restrict__ done) {
    chain_enter();
    if (done != nullptr && *done) return;
    tsqr_root_fix_body(Q, ldq, hq, nc, R, ldr, Rout, ldro);
}

// Down-sweep: for each tile t of TR rows of Q (rows x nc, ldq):
//   Q[tile t] = Q[tile t] * P[t*nc:(t+1)*nc, 0:nc]   (P: ld ldp)
// Body shared by the single and batched kernels: rows [blk*AP_THREADS, ...) of Q, one per
// thread. NC is nc rounded up to the next width there is code for: the FP64 pipe runs every term, so
// padding 10 columns to 16 would cost 60 %.
constexpr int AP_THREADS = 128;

template <int NC>
__device__ void tsqr_apply_body(double* Q, i64 ldq, i64 rows, int nc, int TR, const double* __restrict__ P,
                                i64 ldp, i64 blk, double* p) {
    const i64 r = blk * AP_THREADS + threadIdx.x;
    const i64 t = (blk * AP_THREADS) / TR;   // AP_THREADS divides TR
    // The whole NC x NC tile: the product below runs over NC terms, and entries
    // past nc must be zeros, not whatever an earlier CTA left in shared memory.
    for (int e = threadIdx.x; e < NC * NC; e += AP_THREADS) {
        const int i = e % NC, c = e / NC;
        p[e] = (i < nc && c < nc) ? P[t * nc + i + (i64)c * ldp] : 0.0;
    }
    __syncthreads();
    if (r >= rows) return;   // the last statement of the body: no barrier follows
    double x[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) x[c] = (c < nc) ? Q[r + (i64)c * ldq] : 0.0;
#pragma unroll 2
    for (int c = 0; c < nc; ++c) {
        double y = 0.0;
#pragma unroll
        for (int i = 0; i < NC; ++i) y = fma(x[i], p[i + c * NC], y);
        Q[r + (i64)c * ldq] = y;
    }
}

template <int NC>
__global__ void __launch_bounds__(AP_THREADS)
tsqr_apply_kernel(double* Q, i64 ldq, i64 rows, int nc, int TR, const double* __restrict__ P, i64 ldp,
                  const int* __restrict__ done) {
    __shared__ double p[NC * NC];
    chain_enter();
    if (done != nullptr && *done) return;
    tsqr_apply_body<NC>(Q, ldq, rows, nc, TR, P, ldp, blockIdx.x, p);
}

static int launch_apply(double* Q, i64 ldq, i64 rows, int nc, int TR, const double* P, i64 ldp, const int* done,
                        cudaStream_t st) {
    const unsigned blocks = (unsigned)ceil_div(rows, AP_THREADS);
#define BCGS_APPLY(N) \
    if (nc <= N) { launch_spread(tsqr_apply_kernel<N>, blocks, AP_THREADS, 0, st, Q, ldq, rows, nc, TR, P, ldp, done); break; }
    do {
        BCGS_APPLY(2) BCGS_APPLY(4) BCGS_APPLY(5) BCGS_APPLY(6) BCGS_APPLY(8) BCGS_APPLY(10) BCGS_APPLY(12)
        BCGS_APPLY(14) BCGS_APPLY(16) BCGS_APPLY(20) BCGS_APPLY(24) BCGS_APPLY(28) BCGS_APPLY(32) BCGS_APPLY(40)
        BCGS_APPLY(48) BCGS_APPLY(56) BCGS_APPLY(64)
        return (int)cudaErrorInvalidValue;
    } while (0);
#undef BCGS_APPLY
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

i64 tsqr_workspace_doubles(i64 m, int nc) {
    const int TR = tsqr_tile_rows(nc);
    i64 total = 0, h = m;
    while (h > TR) {
        i64 tiles = ceil_div(h, TR);
        total += tiles * nc * nc;
        h = tiles * nc;
    }
    total += 64 * 64 + 32;                             // + the root tile's R and the checked Cholesky's flag
    const i64 chol = tsqr_check_doubles(nc);           // or its flag and its three blocks
    return total > chol ? total : chol;
}

// The tree from a given level on: level 0 here is (A0, rows0, ld0), factored in
// place; each level's tile R factors are stacked into the next level (in ws),
// until one tile remains (the root). Then the root's signs are fixed, R is
// written to (R, ldR), and the down-sweep brings the explicit Q back to level 0.
template <int NC>
static int tsqr_levels(double* A0, i64 ld0, i64 rows0, int nc, double* R, int ldR, double* ws, const int* done,
                       cudaStream_t st) {
    const int TR = tsqr_tile_rows(nc);
    constexpr int kMaxLevels = 48;   // each level divides the rows by TR / nc >= 2: 2^k rows need at most k levels
    double* lvl_ptr[kMaxLevels];
    i64 lvl_rows[kMaxLevels], lvl_ld[kMaxLevels];
    lvl_ptr[0] = A0;
    lvl_rows[0] = rows0;
    lvl_ld[0] = ld0;
    int L = 0;
    double* cursor = ws;
    while (lvl_rows[L] > TR) {
        if (L + 1 >= kMaxLevels) return (int)cudaErrorInvalidValue;
        const i64 tiles = ceil_div(lvl_rows[L], TR);
        double* next = cursor;
        cursor += tiles * nc * nc;
        const int rc = launch_tiles<NC>(lvl_ptr[L], lvl_ld[L], lvl_rows[L], nc, next, tiles * nc, done, st);
        if (rc) return rc;
        ++L;
        lvl_ptr[L] = next;
        lvl_rows[L] = tiles * nc;
        lvl_ld[L] = tiles * nc;
    }
    // Root: one tile; its R goes to a small slot after the stacks.
    double* rroot = cursor;
    int root_rc = launch_tiles<NC>(lvl_ptr[L], lvl_ld[L], lvl_rows[L], nc, rroot, nc, done, st);
    if (root_rc) return root_rc;
    launch_chained(tsqr_root_fix, 1, 256, 0, st, lvl_ptr[L], lvl_ld[L], (int)lvl_rows[L], nc, rroot, nc, R, ldR, done);
    g_launch_count += 1;
    // Down-sweep.
    for (int l = L - 1; l >= 0; --l) {
        const int rc = launch_apply(lvl_ptr[l], lvl_ld[l], lvl_rows[l], nc, TR, lvl_ptr[l + 1], lvl_ld[l + 1], done, st);
        if (rc) return rc;
    }
    return (int)cudaGetLastError();
}

template <int NC>
static int tsqr_run(double* X, i64 ld, i64 m, int c0, int nc, double* R, int ldR, double* ws,
                    const int* done, cudaStream_t st) {
    return tsqr_levels<NC>(X + (i64)c0 * ld, ld, m, nc, R, ldR, ws, done, st);
}

// Row-sharded TSQR: this rank's rows are the TR-row tiles [t0, t0 + nt) of a
// panel of T tiles. The leaf level runs on the local tiles, writing their R
// factors to `mine` (maxt * nc rows, ld maxt * nc); gather(mine, all) places every
// rank's block in rank order; the blocks are assembled into the global level-1
// stack (T * nc rows, as the one-rank tree has it), whose tree every rank runs;
// the down-sweep of the local tiles then uses this rank's rows of level 1's Q.
// With tiles aligned across ranks, every launch sees the data the one-rank TSQR
// sees, so Q and R are bit-identical to it.
template <int NC>
static int tsqr_sharded_run(double* X, i64 ld, i64 m_local, int c0, int nc, double* R, int ldR, double* ws,
                            const TsqrShard& sh, cudaStream_t st) {
    const int TR = tsqr_tile_rows(nc);
    if (sh.T <= 1) return tsqr_run<NC>(X, ld, m_local, c0, nc, R, ldR, ws, nullptr, st);   // one tile: one rank holds it
    double* panel = X + (i64)c0 * ld;
    const i64 nt = ceil_div(m_local, TR);
    const i64 ldm = sh.maxt * nc;
    if (nt > 0) {
        const int trc = launch_tiles<NC>(panel, ld, m_local, nc, sh.mine, ldm, nullptr, st);
        if (trc) return trc;
    }
    int rc = sh.gather(sh.ctx, sh.mine, sh.all, ldm * nc, st);
    if (rc) return rc;
    double* lvl1 = ws;
    const i64 ld1 = sh.T * nc;
    for (int r = 0; r < sh.size; ++r) {
        if (sh.nt[r] <= 0) continue;
        rc = (int)cudaMemcpy2DAsync(lvl1 + sh.t0[r] * nc, (size_t)ld1 * sizeof(double), sh.all + (i64)r * ldm * nc,
                                    (size_t)ldm * sizeof(double), (size_t)(sh.nt[r] * nc) * sizeof(double), (size_t)nc,
                                    cudaMemcpyDeviceToDevice, st);
        if (rc) return rc;
    }
    rc = tsqr_levels<NC>(lvl1, ld1, ld1, nc, R, ldR, ws + ld1 * nc, nullptr, st);
    if (rc) return rc;
    if (nt > 0) {
        rc = launch_apply(panel, ld, m_local, nc, TR, lvl1 + sh.t0[sh.rank] * nc, ld1, nullptr, st);
        if (rc) return rc;
    }
    return (int)cudaGetLastError();
}

int launch_tsqr_sharded(double* X, i64 ld, i64 m_local, int c0, int nc, double* R, int ldR, double* ws,
                        const TsqrShard& sh, cudaStream_t st) {
    if (nc <= 0) return 0;
    if (nc <= 8) return tsqr_sharded_run<8>(X, ld, m_local, c0, nc, R, ldR, ws, sh, st);
    if (nc <= 16) return tsqr_sharded_run<16>(X, ld, m_local, c0, nc, R, ldR, ws, sh, st);
    if (nc <= 32) return tsqr_sharded_run<32>(X, ld, m_local, c0, nc, R, ldR, ws, sh, st);
    if (nc <= 64) return tsqr_sharded_run<64>(X, ld, m_local, c0, nc, R, ldR, ws, sh, st);
    return (int)cudaErrorInvalidValue;
}

// Cholesky QR twice (Fukaya, Nakatsukasa, Yanagisawa, Yamamoto 2014), if the panel allows
// it: G = V^T V, R1 = chol(G). With D the column norms of V, the computed G and R1 satisfy
// R1^T R1 = V^T V + D E D, |E_ij| of the order of u times the length of the Gram's chains, so
// V R1^{-1} departs from orthonormal by at most || E || || D R1^{-1} ||_F^2. The step that makes R1
// forms that norm (the pivots alone do not bound it: Kahan's matrix has unit columns, large
// pivots and a condition that grows exponentially with its width). Up to
// kCondLimit the departure is about 10^-7 (at most 0.02 with every rounding of a chain of
// 2048 rows against it, at 64 columns), and a second round brings it to roundoff, as the
// tree does. Beyond (or if a pivot is not a positive number) nothing has been written yet,
// and the tree factors the panel; its kernels read the flag and end at once otherwise.
// On the CPU, 592 panels of 8 to 64 columns (Kahan's, I - a triu, graded): the departure is 0.02
// to 6 times u || D R1^{-1} ||_F^2 up to 0.1, and after the second round at most 1.2e-15. Twice
// m nc^2 / 2 products for the upper Gram and as many for the substitution, against some
// 3.5 m nc^2 issued by the tree, a chain of nc reflectors at every level. Measured at
// 4 10^5 x 32: 4.24 ms by the tree, 1.9 ms this way; at 2^19 x 64: 23.7 and 8.5 ms; at 10^5 x 10:
// 213 and 115 us. A panel that fails the test has cost the first Gram (0.5 ms at
// 4 10^5 x 32).
// All panels of more than 16 columns take this; of 8 and more where the caller allows it
// and the tree has at least two levels (below 8 columns its levels are short: 19 us at 4).
constexpr int kCheckedCols = 8;
constexpr double kCondLimit = 1e9;

static int tsqr_checked(double* X, i64 ld, i64 m, int c0, int nc, double* R, int ldR, double* ws, double* part,
                        int num_sms, int* done, cudaStream_t st) {
    const i64 nn = (i64)nc * nc;
    double *G = ws, *R1 = ws + nn, *R2 = ws + 2 * nn;
    for (int pass = 0; pass < 2; ++pass) {
        const int* gate = pass ? done : nullptr;
        int rc = nc <= 32 ? launch_panel_gram(X, ld, m, c0, nc, G, part, num_sms, gate, st)
                          : launch_gram_fp64(X, ld, m, c0, nc, c0, nc, G, nc, part, true, num_sms, st, gate, false);
        StepJob J;
        J.G = G; J.ldg = nc; J.ny = nc; J.T = pass ? R2 : R1;
        if (!pass) { J.ok = done; J.ok_limit = kCondLimit; }
        J.gate = gate;
        if (!rc) rc = launch_step(J, st);
        if (!rc) rc = launch_update_fp64(X, ld, m, 0, 0, c0, nc, nullptr, 0, J.T, nc, true, st, done);
        if (rc) return rc;
    }
    // R = R2 R1 (overwritten by the tree if the flag is not set).
    return launch_rblock(R, ldR, 0, 0, nc, nullptr, 0, nullptr, 0, R1, R2, 0, st);
}

int launch_tsqr(double* X, i64 ld, i64 m, int c0, int nc, double* R, int ldR, double* ws, double* part, int num_sms,
                bool checked, cudaStream_t st) {
    if (nc <= 0) return 0;
    int* done = nullptr;
    if (nc > 16 || (checked && nc >= kCheckedCols && m > TSQR_TR)) {
        done = reinterpret_cast<int*>(ws);
        ws += 32;
        const int rc = tsqr_checked(X, ld, m, c0, nc, R, ldR, ws, part, num_sms, done, st);
        if (rc) return rc;
    }
    if (nc <= 8) return tsqr_run<8>(X, ld, m, c0, nc, R, ldR, ws, done, st);
    if (nc <= 16) return tsqr_run<16>(X, ld, m, c0, nc, R, ldR, ws, done, st);
    if (nc <= 32) return tsqr_run<32>(X, ld, m, c0, nc, R, ldR, ws, done, st);
    if (nc <= 64) return tsqr_run<64>(X, ld, m, c0, nc, R, ldR, ws, done, st);
    return (int)cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// Batched forms (batched.h): tiles of one tree level, root sign fixes and one
// down-sweep level over many panels (nc <= 16, TR = 256), with the single-panel
// bodies.
// ---------------------------------------------------------------------------
template <int W>
__global__ void __launch_bounds__(32 * W)
tsqr_tile_batched(const TsqrTileJob* __restrict__ jobs, const int* __restrict__ prefix, int njobs) {
    extern __shared__ double smem[];
    const int j = batched_job_of(prefix, njobs, blockIdx.x);
    const TsqrTileJob J = jobs[j];
    tsqr_tile_body<16, W>(J.A, J.lda, J.rows, J.nc, J.A, J.lda, J.Rst, J.ldr, blockIdx.x - prefix[j], smem);
}

__global__ void tsqr_root_batched(const TsqrRootJob* __restrict__ jobs) {
    const TsqrRootJob& J = jobs[blockIdx.x];
    tsqr_root_fix_body(J.Q, J.ldq, J.hq, J.nc, J.R, J.ldr, J.Rout, J.ldro);
}

__global__ void __launch_bounds__(AP_THREADS)
tsqr_apply_batched(const TsqrApplyJob* __restrict__ jobs, const int* __restrict__ prefix, int njobs) {
    __shared__ double p[16 * 16];
    const int j = batched_job_of(prefix, njobs, blockIdx.x);
    const TsqrApplyJob J = jobs[j];
    const i64 blk = blockIdx.x - prefix[j];
    if (J.nc <= 4) tsqr_apply_body<4>(J.Q, J.ldq, J.rows, J.nc, J.TR, J.P, J.ldp, blk, p);
    else if (J.nc <= 8) tsqr_apply_body<8>(J.Q, J.ldq, J.rows, J.nc, J.TR, J.P, J.ldp, blk, p);
    else if (J.nc <= 12) tsqr_apply_body<12>(J.Q, J.ldq, J.rows, J.nc, J.TR, J.P, J.ldp, blk, p);
    else tsqr_apply_body<16>(J.Q, J.ldq, J.rows, J.nc, J.TR, J.P, J.ldp, blk, p);
}

// Sets the batched tile kernel's shared-memory limit (outside any stream capture).
int tsqr_tile_batched_prepare() {
    const int bytes = (int)tsqr_tile_smem_bytes(16);
    const int rc = (int)cudaFuncSetAttribute(tsqr_tile_batched<tsqr_many_warps<16>()>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return rc ? rc : (int)cudaFuncSetAttribute(tsqr_tile_batched<tsqr_tile_warps<16>()>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

int launch_tsqr_tile_batched(const TsqrTileJob* jobs, const int* prefix, int njobs, int items, int ncmax,
                             cudaStream_t st) {
    if (items <= 0) return 0;
    if (ncmax > 16) return (int)cudaErrorInvalidValue;
    const size_t smem = tsqr_tile_smem_bytes(16);
    constexpr int W = tsqr_tile_warps<16>(), WM = tsqr_many_warps<16>();
    if (items >= tsqr_many_tiles<16>())
        tsqr_tile_batched<WM><<<(unsigned)items, 32 * WM, smem, st>>>(jobs, prefix, njobs);
    else
        tsqr_tile_batched<W><<<(unsigned)items, 32 * W, smem, st>>>(jobs, prefix, njobs);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

int launch_tsqr_root_batched(const TsqrRootJob* jobs, int njobs, cudaStream_t st) {
    if (njobs <= 0) return 0;
    tsqr_root_batched<<<(unsigned)njobs, 256, 0, st>>>(jobs);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

int launch_tsqr_apply_batched(const TsqrApplyJob* jobs, const int* prefix, int njobs, int items, int ncmax,
                              cudaStream_t st) {
    if (items <= 0) return 0;
    if (ncmax > 16) return (int)cudaErrorInvalidValue;
    tsqr_apply_batched<<<(unsigned)items, AP_THREADS, 0, st>>>(jobs, prefix, njobs);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

}  // namespace bcgs
