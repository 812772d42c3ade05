// Small FP64 block kernels of the BCGS step (s <= 64), run between the tall passes
// on the reduced Gram blocks.
//
//   step   : everything a block step computes on the reduced Gram G in one launch:
//            T = chol(Om_Y - Y^T Y)                        (SRC/orth.c:200-204, ...)
//            the next block's S = [Z ; T^{-T}(G_mid - Y^T Z)]   (:155-159, :310-314)
//            Sd = chol(Om_Z - S^T S)                       (:160-171)
//            and the R column block of the current step    (:211-215, :356-360)
//   rblock : the R column block alone (the variants whose factors come from TSQR)
//
// One elimination. With Y = G[0:K, 0:ny] and Z = G[0:K, ny:ny+nz] the three
// factorizations above are one upper Cholesky factorization
//     U^T U = G[K:K+N, 0:N] - [Y Z]^T [Y Z],   U = [T  S_mid ; 0  Sd],  N = ny + nz,
// so they run as N right-looking steps on one N x N matrix in shared memory, and
// carrying the identity along gives U^{-1}, which the tensor-core update's factor is
// built from ([Q U X] times [-G U^{-1} ; U^{-1}]).
//
// What bounds it. An FP64 instruction of one warp occupies its quarter of the SM for
// 64 clocks, however many lanes are active, and returns after as many: there is no
// latency left to hide, only instructions to save (a square root costs 600 clocks, a
// division 570). So the K N^2 / 2 products of [Y Z]^T [Y Z] are spread over the CTAs of
// a cluster (kGroups row groups, summed per group and then over the groups through
// distributed shared memory in a fixed order). The elimination, a chain of N
// dependent steps, runs on one CTA: in step j, warp 0 finishes row j + 1 and makes it
// the next pivot row (five dependent instructions) while the other warps update the
// rows below, eight lanes a row because the rows are short.
// One launch replaces four per block step. Measured per step, K = 240: 65 us before
// (two Choleskys, S, R block) and 18.5 us now at N = 20; 145 and 31 us at N = 32; 1850
// and 430 us at N = 128, where the elimination fills its SM (N^3 / 3 multiply-adds,
// 270 us of it).
// The arithmetic does not depend on the number of CTAs per job, so the batched
// launches (one CTA per matrix when there are many) give the single launch's bits.
#include "batched.h"
#include "common.cuh"
#include "kernels.h"

#include <cooperative_groups.h>

namespace bcgs {

namespace cg = cooperative_groups;

namespace {
constexpr int ST_THREADS = 256;
constexpr int ST_WARPS = ST_THREADS / 32;
constexpr int SMAX = 64;
constexpr int kGroups = 8;      // row groups of [Y Z]^T [Y Z]
constexpr int kTileRows = 32;   // rows of [Y Z] staged at a time

// Entry e of the upper trapezoid (rows r < nr, columns r <= c < n), column by column.
__device__ __forceinline__ void trap_rc(int e, int nr, int& r, int& c) {
    const int tri = nr * (nr + 1) / 2;
    if (e < tri) {
        c = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
        while ((c + 1) * (c + 2) / 2 <= e) ++c;
        while (c * (c + 1) / 2 > e) --c;
        r = e - c * (c + 1) / 2;
    } else {
        const int f = e - tri;
        c = nr + f / nr;
        r = f - (c - nr) * nr;
    }
}
__host__ __device__ inline int trap_size(int nr, int n) { return nr * (nr + 1) / 2 + (n - nr) * nr; }
}  // namespace

// Shared memory of one CTA (doubles): the N x N matrix (also the staging tile of the
// products and Sd of the R block), the sums of this CTA's row groups (later Sold),
// and the pivots.
__host__ __device__ inline int step_matrix_doubles(int n) { return (n > kTileRows ? n : kTileRows) * (n + 1); }
__host__ __device__ inline int step_sums_doubles(int n, int ny, int ctas) {
    const int sums = (kGroups / ctas) * trap_size(n, n);
    return sums > ny * ny ? sums : ny * ny;   // Sold moves in when the sums have been used
}
static size_t step_smem_bytes(int n, int ny, int ctas) {
    return (size_t)(step_matrix_doubles(n) + step_sums_doubles(n, ny, ctas) + 4 * n + 2) * sizeof(double);
}

// R[0:K, c0:c0+ny] = A + Y Sd_old (mode 0) or A + Y (mode 1), rows [r0, r1), as
// thread t0 of nt. sd: ny x ny, ld ny, upper (mode 0).
__device__ __forceinline__ void r_rows(double* R, int ldR, int c0, int ny, const double* A, int lda, const double* B,
                                       int ldb, const double* sd, int mode, int r0, int r1, int t0, int nt) {
    const int rows = r1 - r0;
    for (int e = t0; e < rows * ny; e += nt) {
        const int i = r0 + e % rows, j = e / rows;
        double v = __ldg(A + i + (i64)j * lda);
        if (mode == 0) {
            double t = 0.0;
            for (int l = 0; l <= j; ++l) t = fma(__ldg(B + i + (i64)l * ldb), sd[l + j * ny], t);
            v += t;
        } else {
            v += __ldg(B + i + (i64)j * ldb);
        }
        R[i + (i64)(c0 + j) * ldR] = v;
    }
}

// R[c0:c0+ny, c0:c0+ny] = Yd Sd (mode 0) or upper(Yd) on the upper part (mode 1),
// Yd(i, l) = yd[i * yi + l * yl].
__device__ __forceinline__ void r_diag(double* R, int ldR, int c0, int ny, const double* yd, int yi, int yl,
                                       const double* sd, int mode) {
    for (int e = threadIdx.x; e < ny * ny; e += blockDim.x) {
        const int i = e % ny, j = e / ny;
        double* dst = R + (c0 + i) + (i64)(c0 + j) * ldR;
        if (mode == 0) {
            double t = 0.0;
            if (i <= j)
                for (int l = i; l <= j; ++l) t = fma(yd[i * yi + l * yl], sd[l + j * ny], t);
            *dst = t;
        } else if (i <= j) {
            *dst = yd[i * yi + j * yl];
        }
    }
}

// Entry e of the right-hand side: G[K + r, c] minus the groups' sums, group by group
// in a fixed tree. (Not for the entries of a breakdown: see the end of step_body.)
template <int C>
__device__ __forceinline__ double step_entry(const StepJob& J, int r, int c, int e, int E, double* gs) {
    double g[kGroups];
#pragma unroll
    for (int k = 0; k < kGroups; ++k) {
        constexpr int PER = kGroups / C;
        double* base = gs;
        if constexpr (C > 1) base = cg::this_cluster().map_shared_rank(gs, k / PER);
        g[k] = base[(k % PER) * E + e];
    }
    return __ldg(J.G + (J.K + r) + (i64)c * J.ldg) -
           (((g[0] + g[1]) + (g[2] + g[3])) + ((g[4] + g[5]) + (g[6] + g[7])));
}

// One job by a cluster of C CTAs (rank = this CTA's), C | kGroups. PANEL: of a checked TSQR
// panel (J.ok, J.gate), in code of its own so that the other steps carry none of it.
template <int C, bool PANEL = false>
__device__ void step_body(const StepJob& J, int rank, double* sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ny = J.ny, nz = J.nz, n = ny + nz;
    const int nr = (nz > 0 && !J.scaled) ? ny : n;   // pivots
    const int ld = n + 1;
    const int E = trap_size(nr, n);
    double* a = sm;
    double* gs = sm + step_matrix_doubles(n);
    double* s_u = gs + step_sums_doubles(n, ny, C);   // pivots of U and their reciprocals
    double* s_t = s_u + 2 * n;                        // the pivot row over the pivot, two slots
    int* s_stop = reinterpret_cast<int*>(s_t + 2 * n);   // and whether it cannot be used

    // ---- products: one sum per row group and entry, rows in order. The rows of this
    // CTA's groups are staged in tiles that may span groups; a sum goes on from
    // where the previous tile left it, so it does not depend on the tiling. ----
    constexpr int PER = kGroups / C;
    const int L = (((J.K + kGroups - 1) / kGroups) + 3) & ~3;
    const int k0 = min(J.K, rank * PER * L), k1 = min(J.K, (rank + 1) * PER * L);
    for (int e = tid; e < PER * E; e += ST_THREADS) gs[e] = 0.0;
#pragma unroll 1
    for (int t0 = k0; t0 < k1; t0 += kTileRows) {
        const int t1 = min(k1, t0 + kTileRows);
        for (int e = tid; e < kTileRows * n; e += ST_THREADS) {
            const int rr = e % kTileRows, c = e / kTileRows;
            if (t0 + rr < t1) a[rr * ld + c] = J.G[t0 + rr + (i64)c * J.ldg];
        }
        __syncthreads();
        const int q0 = (t0 - k0) / L, q1 = (t1 - 1 - k0) / L;   // groups with rows in this tile
        for (int w = tid; w < (q1 - q0 + 1) * E; w += ST_THREADS) {
            const int q = q0 + w / E, e = w % E;
            int r, c;
            trap_rc(e, nr, r, c);
            const int i0 = max(0, k0 + q * L - t0), i1 = min(t1, k0 + (q + 1) * L) - t0;
            double acc = gs[q * E + e];
            const double* x = a + r;
            const double* y = a + c;
#pragma unroll 4
            for (int i = i0; i < i1; ++i) acc = fma(x[i * ld], y[i * ld], acc);
            gs[q * E + e] = acc;
        }
        __syncthreads();
    }
    __syncthreads();
    if constexpr (C > 1) cg::this_cluster().sync();

    // ---- S_top = Z, and the R block's rows of Q, by the CTAs that do not eliminate ----
    if (C == 1 || rank > 0) {
        const int nt = (C == 1 ? 1 : C - 1) * ST_THREADS;
        const int t = (C == 1 ? 0 : rank - 1) * ST_THREADS + tid;
        if (J.S != nullptr)
            for (int e = t; e < J.K * nz; e += nt) {
                const int i = e % J.K, j = e / J.K;
                J.S[i + (i64)j * (J.K + ny)] = __ldg(J.G + i + (i64)(ny + j) * J.ldg);
            }
        if (J.mode >= 0) {
            if (J.mode == 0)
                for (int e = tid; e < ny * ny; e += ST_THREADS) {
                    const int i = e % ny, j = e / ny;
                    a[i + j * ny] = i <= j ? __ldg(J.Sold + i + (i64)j * ny) : 0.0;
                }
            __syncthreads();
            r_rows(J.R, J.ldR, J.c0, ny, J.A, J.lda, J.G, J.ldg, a, J.mode, 0, J.K, t, nt);
            __syncthreads();
        }
    }
    if constexpr (C > 1) {
        if (rank > 0) {
            // This CTA's sums stay readable until rank 0 has fetched them.
            cg::this_cluster().sync();
            return;
        }
    }

    // This CTA's part of Sold, for the diagonal block at the end.
    double sold[SMAX * SMAX / ST_THREADS];
#pragma unroll
    for (int k = 0; k < SMAX * SMAX / ST_THREADS; ++k) {
        const int e = tid + k * ST_THREADS;
        sold[k] = J.mode == 0 && e < ny * ny && e % ny <= e / ny ? J.Sold[e] : 0.0;
    }

    // ---- elimination: main part in the upper triangle (diagonal included), the
    // carried identity's strictly lower part below it (its unit diagonal implied) ----
    for (int e = tid; e < E; e += ST_THREADS) {
        int r, c;
        trap_rc(e, nr, r, c);
        a[r * ld + c] = step_entry<C>(J, r, c, e, E, gs);
    }
    for (int e = tid; e < n * n; e += ST_THREADS) {
        const int r = e / n, c = e % n;
        if (c < r) a[r * ld + c] = 0.0;
        if (r >= nr && c >= r) a[r * ld + c] = c == r ? 1.0 : 0.0;   // rows that are not eliminated
    }
    __syncthreads();
    // Warp 0: row r becomes the pivot row. Its pivot's reciprocal and the row over the
    // pivot go to slot r & 1 (the carried identity has 1 at c = r). A pivot that is
    // not a positive number of ordinary size ends the fast path (an integer test: a
    // comparison would be one more FP64 instruction).
    const bool carry = J.Uinv != nullptr || (PANEL && J.ok != nullptr);
    // (Loops over the columns are kept rolled: an FP64 instruction that is only
    // predicated off still takes its 64 clocks.)
    auto publish = [&](int r, double d, double x0) {
        const double inv = recip(d);
        const unsigned hi = (unsigned)__double2hiint(d);
        if (lane == 0) s_stop[r & 1] = !(hi >= 0x05D00000u && hi < 0x7A100000u);   // 2^-930 .. 2^930
        double* t = s_t + (r & 1) * n;
        if (n <= 32) {
            const double y = x0 * inv;
            if (lane < n) t[lane] = lane == r ? inv : y;
            return;
        }
#pragma unroll 1
        for (int c = carry ? lane : (r & ~31) + lane; c < n; c += 32) {
            const double y = a[r * ld + c] * inv;
            t[c] = c == r ? inv : y;
        }
    };
    if (warp == 0) publish(0, a[0], lane < n ? a[lane] : 0.0);
    __syncthreads();
    // Workers: eight lanes a row, four rows a warp, the warps of warp 0's quarter last.
    const int slot = warp == 0 ? -1 : (warp == 4 ? 6 : (warp > 4 ? warp - 2 : warp - 1)) * 4 + (lane >> 3);
    const int l8 = lane & 7;
    bool fast = s_stop[0] == 0;
    int stop = 0;   // the pivot that ended the fast path
    for (int j = 0; j < nr && fast; ++j) {
        const double* pr = a + j * ld;
        const double* t = s_t + (j & 1) * n;
        if (warp == 0) {
            const int r = j + 1;
            if (r < n) {
                double* row = a + r * ld;
                const double f = -pr[r];
                if (n <= 32) {
                    const int c = min(lane, n - 1);
                    const double x = row[c], y = fma(f, t[c], x);
                    const double z = (c <= j ? carry : r < nr) ? y : x;
                    if (lane < n) row[lane] = z;
                    if (r < nr) publish(r, __shfl_sync(0xffffffffu, z, r), z);
                } else {
#pragma unroll 1
                    for (int c = carry ? lane : (r & ~31) + lane; c < n; c += 32) {
                        const double x = row[c], y = fma(f, t[c], x);
                        row[c] = (c <= j ? carry : r < nr) ? y : x;
                    }
                    __syncwarp();
                    if (r < nr) publish(r, row[r], 0.0);
                }
            }
        } else {
            const int na = carry ? j + 1 : 0;   // carried columns of every row
            for (int r = j + 2 + slot; r < n; r += 4 * (ST_WARPS - 1)) {
                double* row = a + r * ld;
                const double f = -pr[r];
                const int len = na + (r < nr ? n - r : 0);
                int q = l8, c = q < na ? q : r + q - na;
                double x = q < len ? row[c] : 0.0, y = q < len ? t[c] : 0.0;
#pragma unroll 1
                while (q < len) {
                    const int q1 = q + 8, c1 = q1 < na ? q1 : r + q1 - na;
                    double x1 = 0.0, y1 = 0.0;
                    if (q1 < len) { x1 = row[c1]; y1 = t[c1]; }
                    row[c] = fma(f, y, x);
                    q = q1; c = c1; x = x1; y = y1;
                }
            }
        }
        __syncthreads();
        // Slot (j + 1) & 1 is next written after the barrier that ends step j + 1.
        stop = j + 1;
        if (stop < nr) fast = s_stop[stop & 1] == 0;
    }

    if (fast) {
        // Row r of U is the eliminated row over the square root of its pivot; the
        // carried rows scale the same way and give U^{-T}.
        for (int r = tid; r < n; r += ST_THREADS) {
            const double d = r < nr ? a[r * ld + r] : 1.0, v = rsqrt(d);
            s_u[r] = root(d, v);
            s_u[n + r] = v;
        }
        __syncthreads();
        for (int r = warp; r < n; r += ST_WARPS) {
            const double v = s_u[n + r];
            for (int c = lane; c < n; c += 32) {
                const double x = c == r ? s_u[r] : a[r * ld + c] * v;
                a[r * ld + c] = x;
                if (r < ny && c < ny) J.T[r + (i64)c * ny] = c >= r ? x : 0.0;
                else if (r < ny) J.S[(J.K + r) + (i64)(c - ny) * (J.K + ny)] = x;
                else if (c >= ny && J.scaled) J.Sd[(r - ny) + (i64)(c - ny) * nz] = c >= r ? x : 0.0;
                if (J.Uinv != nullptr) J.Uinv[c + (i64)r * n] = c < r ? x : (c == r ? v : 0.0);
            }
        }
        __syncthreads();
        if (PANEL && J.ok != nullptr) {
            // Row r of a's lower part is row r of U^{-T}: the sum of G_cc (U^{-T})_rc^2, in a
            // fixed order. (A sum that is Inf or NaN is not within the limit.)
            __shared__ double s_norm[ST_WARPS];
            double p = 0.0;
            for (int r = warp; r < n; r += ST_WARPS)
                for (int c = lane; c <= r; c += 32) {
                    const double x = c == r ? s_u[n + r] : a[r * ld + c];
                    p = fma(x * x, __ldg(J.G + c + (i64)c * J.ldg), p);
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
            if (lane == 0) s_norm[warp] = p;
            __syncthreads();
            if (tid == 0) {
                for (int w = 1; w < ST_WARPS; ++w) p += s_norm[w];
                *J.ok = p <= J.ok_limit;
            }
        }
    } else if (PANEL && J.ok != nullptr) {
        if (tid == 0) *J.ok = 0;
    } else {
        // A pivot out of range: the same factorization by dot products. At a
        // breakdown (a pivot <= 0) the factor keeps the rows before it, and the rows
        // from it on hold the matrix that was to be factored, as dpotrf leaves
        // them; what follows goes on with that factor. Not a path for speed.
        // The right-hand side is formed anew, each entry one chain that starts at G's:
        // where a column is noise next to those before it, G minus a rounded sum is a
        // small multiple of G's last bit, often 0, and dividing by that pivot would
        // end in Inf and NaN; the chain keeps the products' lower bits. A pivot <= 0 of either
        // form is reported: that of the rounded sums is the reference's (dgemm, then dpotrf).
        int bad = a[stop * ld + stop] <= 0.0 ? stop + 1 : 0;   // 1-based pivot (thread 0's counts)
        __syncthreads();
        for (int e = tid; e < E; e += ST_THREADS) {
            int r, c;
            trap_rc(e, nr, r, c);
            const double* x = J.G + (i64)r * J.ldg;
            const double* y = J.G + (i64)c * J.ldg;
            double v = __ldg(y + J.K + r);
#pragma unroll 4
            for (int l = 0; l < J.K; ++l) v = fma(-__ldg(x + l), __ldg(y + l), v);
            a[r * ld + c] = v;
        }
        for (int e = tid; e < n * n; e += ST_THREADS) {
            const int r = e / n, c = e % n;
            if (c < r) a[r * ld + c] = 0.0;
            if (r >= nr && c >= r) a[r * ld + c] = c == r ? 1.0 : 0.0;
        }
        __syncthreads();
        // Upper Cholesky of rows and columns [o, o + k), up to a breakdown.
        auto chol = [&](int o, int k) {
            for (int j = o; j < o + k; ++j) {
                __syncthreads();
                if (tid == 0) {
                    double d = a[j * ld + j];
                    for (int i = o; i < j; ++i) d = fma(-a[i * ld + j], a[i * ld + j], d);
                    s_stop[0] = d <= 0.0;
                    a[j * ld + j] = d <= 0.0 ? d : sqrt(d);
                    if (d <= 0.0 && (bad == 0 || j < bad)) bad = j + 1;
                }
                __syncthreads();
                if (s_stop[0] != 0) break;
                for (int c = j + 1 + tid; c < o + k; c += ST_THREADS) {
                    double v = a[j * ld + c];
                    for (int i = o; i < j; ++i) v = fma(-a[i * ld + j], a[i * ld + c], v);
                    a[j * ld + c] = v / a[j * ld + j];
                }
            }
            __syncthreads();
        };
        chol(0, ny);
        // S_mid = T^{-T} (G_mid - Y^T Z), one column per thread.
        for (int c = ny + tid; c < n; c += ST_THREADS)
            for (int i = 0; i < ny; ++i) {
                double v = a[i * ld + c];
                for (int l = 0; l < i; ++l) v = fma(-a[l * ld + i], a[l * ld + c], v);
                a[i * ld + c] = v / a[i * ld + i];
            }
        __syncthreads();
        if (nr > ny) {
            for (int e = tid; e < nz * nz; e += ST_THREADS) {
                const int r = ny + e % nz, c = ny + e / nz;
                if (r > c) continue;
                double v = a[r * ld + c];
                for (int l = 0; l < ny; ++l) v = fma(-a[l * ld + r], a[l * ld + c], v);
                a[r * ld + c] = v;
            }
            chol(ny, nz);
        }
        if (tid == 0 && bad != 0 && J.status != nullptr && J.status[0] == 0) {
            J.status[0] = J.step + (bad > ny ? 1 : 0);
            J.status[1] = bad > ny ? bad - ny : bad;
        }
        for (int e = tid; e < n * n; e += ST_THREADS) {
            const int r = e / n, c = e % n;
            const double x = a[r * ld + c];
            if (r < ny && c < ny) J.T[r + (i64)c * ny] = x;
            else if (r < ny) J.S[(J.K + r) + (i64)(c - ny) * (J.K + ny)] = x;
            else if (c >= ny && J.scaled) J.Sd[(r - ny) + (i64)(c - ny) * nz] = x;
        }
        if (J.Uinv != nullptr) {
            // Column c of U^{-1} by back substitution, through global memory.
            for (int c = tid; c < n; c += ST_THREADS) {
                double* y = J.Uinv + (i64)c * n;
                for (int i = n - 1; i >= 0; --i) {
                    double v = i == c ? 1.0 : 0.0;
                    for (int l = i + 1; l <= c; ++l) v = fma(-a[i * ld + l], y[l], v);
                    y[i] = i <= c ? v / a[i * ld + i] : 0.0;
                }
            }
        }
        __syncthreads();
    }
    if (J.mode >= 0) {
        // a's leading block is T (row by row) on either path; the sums are done with.
#pragma unroll
        for (int k = 0; k < SMAX * SMAX / ST_THREADS; ++k)
            if (tid + k * ST_THREADS < ny * ny) gs[tid + k * ST_THREADS] = sold[k];
        __syncthreads();
        r_diag(J.R, J.ldR, J.c0, ny, a, ld, 1, gs, J.mode);
    }
    if constexpr (C > 1) cg::this_cluster().sync();
}

// CTAs per SM given so that the registers come out as they are fastest. The cluster of eight
// is left to the compiler (64 registers; with 112 bcgsi2P1s split at 2^19 x 512, s = 64,
// 34.6 -> 34.7 ms); the others would be spilled to 64 or 80 (a batch of 96 in the split form
// 10.59 -> 10.63 ms), except the batched form with many jobs, three of whose CTAs share an SM.
template <int C>
__global__ void __launch_bounds__(ST_THREADS, C == 8 ? 0 : 1) step_kernel(const __grid_constant__ StepJob job) {
    extern __shared__ double sm[];
    chain_enter();
    step_body<C>(job, C == 1 ? 0 : (int)blockIdx.x, sm);
}

__global__ void __launch_bounds__(ST_THREADS, 1) step_panel_kernel(const __grid_constant__ StepJob job) {
    extern __shared__ double sm[];
    chain_enter();
    if (job.gate != nullptr && *job.gate == 0) return;
    step_body<1, true>(job, 0, sm);
}

// Batched form: CTAs [b C, (b + 1) C) run job b.
template <int C>
__global__ void __launch_bounds__(ST_THREADS, C == 1 ? 3 : 1) step_batched(const StepJob* __restrict__ jobs) {
    extern __shared__ double sm[];
    const StepJob J = jobs[blockIdx.x / C];
    step_body<C>(J, (int)(blockIdx.x % C), sm);
}

// The R column block alone: K x ny rows of Q by 32-row CTAs, the diagonal block by
// the last CTA.
__global__ void __launch_bounds__(ST_THREADS)
rblock_kernel(double* R, int ldR, int c0, int K, int ny, const double* A, int lda, const double* B, int ldb,
              const double* Sd, const double* Yd, int mode) {
    __shared__ double sd[SMAX * SMAX];
    chain_enter();
    if ((int)blockIdx.x == (int)gridDim.x - 1) {
        r_diag(R, ldR, c0, ny, Yd, 1, ny, Sd, mode);
        return;
    }
    if (mode == 0)
        for (int e = threadIdx.x; e < ny * ny; e += blockDim.x) {
            const int i = e % ny, j = e / ny;
            sd[i + j * ny] = (i <= j) ? Sd[i + (i64)j * ny] : 0.0;
        }
    __syncthreads();
    const int r0 = (int)blockIdx.x * 32;
    r_rows(R, ldR, c0, ny, A, lda, B, ldb, sd, mode, r0, min(K, r0 + 32), threadIdx.x, blockDim.x);
}

namespace {

template <class K>
int launch_clustered(K kernel, unsigned grid, int ctas, size_t smem, bool chained, cudaStream_t st, void** args) {
    const int rc = smem > 48 * 1024 ? smem_attr((const void*)kernel, (int)smem) : 0;
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(ST_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int na = 0;
    if (chained) {   // as launch_chained
        at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (ctas > 1) {
        at[na].id = cudaLaunchAttributeClusterDimension;
        at[na].val.clusterDim.x = (unsigned)ctas;
        at[na].val.clusterDim.y = 1;
        at[na++].val.clusterDim.z = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = na;
    const cudaError_t ce = cudaLaunchKernelExC(&cfg, (const void*)kernel, args);
    g_launch_count += 1;
    return (int)(ce != cudaSuccess ? ce : cudaGetLastError());
}

bool step_valid(const StepJob& J) {
    return J.ny >= 1 && J.ny <= SMAX && J.nz >= 0 && J.nz <= SMAX && J.K >= 0 && J.G != nullptr && J.T != nullptr &&
           (J.nz == 0 || J.S != nullptr) && (!J.scaled || J.nz == 0 || J.Sd != nullptr) &&
           ((J.ok == nullptr && J.gate == nullptr) || (J.K == 0 && J.nz == 0));
}

}  // namespace

// CTAs per job: a cluster of 8 once the products take longer on one CTA (two
// multiply-adds per clock, the rows in one tile) than the cluster's barriers and
// remote reads, about 2 us.
int launch_step(const StepJob& J, cudaStream_t st) {
    if (!step_valid(J)) return (int)cudaErrorInvalidValue;
    const int n = J.ny + J.nz;
    void* args[1] = {const_cast<StepJob*>(&J)};
    if (J.ok != nullptr || J.gate != nullptr)
        return launch_clustered(step_panel_kernel, 1, 1, step_smem_bytes(n, J.ny, 1), true, st, args);
    if (J.K <= kTileRows && (i64)trap_size(n, n) * J.K <= 8192)
        return launch_clustered(step_kernel<1>, 1, 1, step_smem_bytes(n, J.ny, 1), true, st, args);
    return launch_clustered(step_kernel<8>, 8, 8, step_smem_bytes(n, J.ny, 8), true, st, args);
}

// Batched: enough CTAs per job to spread a small batch over the SMs; one each once the
// jobs alone fill them. Shared memory for the widest job a batch of blocks of up to 16
// columns can have.
int launch_step_batched(const StepJob* jobs, int njobs, cudaStream_t st) {
    if (njobs <= 0) return 0;
    constexpr int N = 32, NY = 16;
    void* args[1] = {(void*)&jobs};
    auto launch = [&](auto kernel, int ctas) {
        return launch_clustered(kernel, (unsigned)(njobs * ctas), ctas, step_smem_bytes(N, NY, ctas), false, st, args);
    };
    if (njobs <= 64) return launch(step_batched<8>, 8);
    if (njobs <= 512) return launch(step_batched<2>, 2);
    return launch(step_batched<1>, 1);
}

int launch_rblock(double* R, int ldR, int c0, int K, int ny, const double* A, int lda, const double* B, int ldb,
                  const double* Sd, const double* Yd, int mode, cudaStream_t st) {
    if (ny <= 0) return 0;
    if (ny > SMAX) return (int)cudaErrorInvalidValue;
    launch_chained(rblock_kernel, (unsigned)((K + 31) / 32 + 1), ST_THREADS, 0, st, R, ldR, c0, K, ny, A, lda, B, ldb, Sd, Yd,
                                                                        mode);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

}  // namespace bcgs
