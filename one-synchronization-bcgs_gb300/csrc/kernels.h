// Internal launcher declarations shared by the kernel files and the C-ABI layer.
// All matrices are column-major FP64 device buffers; every launcher enqueues on
// `st` and returns a cudaError_t value (0 on success).
#pragma once

#include <atomic>

#include <cuda_runtime.h>

namespace bcgs {

using i64 = long long;

// Number of kernels enqueued by the launchers below since load (host counter;
// split-precision batches enqueue from several host threads).
extern std::atomic<long long> g_launch_count;
// Number of launches of the fixed-order Gram reduction (the kernel that stands
// in for each MPI_Allreduce of the reference).
extern std::atomic<long long> g_reduce_count;

// bytes of zeros at p, by a kernel on st (not a copy-engine memset). Counted in
// g_launch_count and also in g_aux_launch_count, which the per-class profile
// subtracts so that its launch counts are those of the classes' own kernels.
int zero_async(void* p, size_t bytes, cudaStream_t st);
extern std::atomic<long long> g_aux_launch_count;

// Raises kernel fn's dynamic shared-memory limit to `bytes` on the current
// device, once per (device, kernel). Call outside any stream capture.
int smem_attr(const void* fn, int bytes);

// C (na x nb, ld ldo) = X[:, a0:a0+na]^T X[:, b0:b0+nb] over m rows, FP64, with a
// fixed-order two-stage reduction through `part` (gram_part_doubles_fp64 doubles).
// upper_only: only the entries on or above the diagonal of X^T X are defined. gate: if
// not null and *gate is 0, the product is left out (out is then undefined). counted:
// whether this is one of the algorithm's synchronizations (g_reduce_count).
i64 gram_part_doubles_fp64(i64 m, int na_max, int nb_max);   // for any na, nb up to these
// Rows per chunk forced by orth_gb300_set_gram_chunk_rows (0: default policy).
extern long long g_gram_chunk_rows;
int launch_gram_fp64(const double* X, i64 ld, i64 m, int a0, int na, int b0, int nb,
                     double* out, int ldo, double* part, bool upper_only, int num_sms, cudaStream_t st,
                     const int* gate = nullptr, bool counted = true);

// out (na x nb, ld ldo) = fixed-order sum of nchunks partials part[c][i + j*na].
int launch_gram_reduce(const double* part, int nchunks, int na, int nb, double* out, int ldo,
                       cudaStream_t st);
int gram_reduce_ctas(int na, int nb);   // CTAs of one reduction
// The same sum in another fixed order, with a shorter chain. counted: as launch_gram_fp64.
int launch_gram_reduce_sliced(const double* part, int nchunks, int na, int nb, double* out, int ldo, bool counted,
                              cudaStream_t st);
int gram_reduce_sliced_ctas(int na, int nb);

// X[:, c0:c0+nc] = (X[:, c0:c0+nc] - X[:, q0:q0+K] S) T^{-1}; T upper (nc x nc) or null.
// any_split: K may be summed in quarters, by a rule on m; without it each row's result
// does not depend on how many rows there are (the row-sharded path). gate: if not null
// and *gate is 0, X is left as it is.
int launch_update_fp64(double* X, i64 ld, i64 m, int q0, int K, int c0, int nc,
                       const double* S, int lds, const double* T, int ldt, bool any_split, cudaStream_t st,
                       const int* gate = nullptr);

// The small work of one block step on the reduced Gram G (small_fp64.cu): with
// Y = G[0:K, 0:ny], Z = G[0:K, ny:ny+nz],
//   T = chol(G[K:K+ny, 0:ny] - Y^T Y)                     (ny x ny, ld ny, lower part 0)
// and, if nz > 0, the next block's first pass
//   S = [Z ; T^{-T} (G[K:K+ny, ny:] - Y^T Z)]             ((K + ny) x nz, ld K + ny)
//   Sd = chol(G[K+ny:, ny:] - S^T S), if scaled           (nz x nz, ld nz)
// and, if mode >= 0, the R column block at columns [c0, c0 + ny): A + Y Sold above
// the diagonal block T Sold (mode 0; Sold ny x ny, ld ny), or A + Y above upper(T)
// (mode 1). Sold and A may be an earlier step's Sd and S but not this job's.
// Uinv (may be null), (ny+nz) x (ny+nz): the inverse of U = [T S_mid ; 0 Sd] (Sd = I
// if not scaled). A breakdown of T is recorded in status as block step `step`, one
// of Sd as step + 1. ny, nz <= 64.
struct StepJob {
    const double* G = nullptr;
    int ldg = 0, K = 0, ny = 0, nz = 0, scaled = 0, step = 0;
    double *T = nullptr, *S = nullptr, *Sd = nullptr, *Uinv = nullptr;
    int* status = nullptr;
    int mode = -1, c0 = 0, ldR = 0, lda = 0;
    double* R = nullptr;
    const double *A = nullptr, *Sold = nullptr;
    // If not null (K = 0, nz = 0): *ok = || D T^{-1} ||_F^2 <= ok_limit, D the square roots of
    // G's diagonal: the squared condition of the columns behind G, each scaled to norm 1.
    // T is only defined if it is.
    int* ok = nullptr;
    double ok_limit = 0.0;
    const int* gate = nullptr;   // K = 0, nz = 0: if not null and *gate is 0, nothing is done
};
int launch_step(const StepJob& J, cudaStream_t st);
// One job per matrix, ny and nz at most 16 each.
int launch_step_batched(const StepJob* jobs, int njobs, cudaStream_t st);

// R[0:K, c0:c0+ny] = A + B Sd and R[c0:c0+ny, c0:] = Yd Sd (mode 0; Sd, Yd ny x ny,
// upper, ld ny), or A + B and upper(Yd) (mode 1).
int launch_rblock(double* R, int ldR, int c0, int K, int ny, const double* A, int lda,
                  const double* B, int ldb, const double* Sd, const double* Yd, int mode, cudaStream_t st);

// Upper Gram (nc x nc, ld nc) of X[:, c0:c0+nc], nc <= 32, through part, which holds
// panel_gram_part_doubles(m, s) for panels of up to s columns (the rows forced by
// g_gram_chunk_rows play no part); gate as launch_gram_fp64.
i64 panel_gram_part_doubles(i64 m, int s);
int launch_panel_gram(const double* X, i64 ld, i64 m, int c0, int nc, double* G, double* part, int num_sms,
                      const int* gate, cudaStream_t st);

// Explicit TSQR of X[:, c0:c0+nc] in place; R (nc x nc, ldR) upper with diag >= 0.
int tsqr_tile_rows(int nc);
i64 tsqr_workspace_doubles(i64 m, int nc);
// part: panel_gram_part_doubles(m, nc) doubles, or gram_part_doubles_fp64(m, nc, nc) for more
// than 32 columns; only written before the tree runs, so it may lie in ws from
// tsqr_check_doubles(nc) on. checked: panels of up to 16 columns may take Cholesky QR
// too (not in BCGSI+P-1S, whose batched plans use the tree).
inline i64 tsqr_check_doubles(int nc) { return 32 + 3LL * nc * nc; }   // the checked Cholesky's flag and blocks in ws
int launch_tsqr(double* X, i64 ld, i64 m, int c0, int nc, double* R, int ldR, double* ws, double* part, int num_sms,
                bool checked, cudaStream_t st);

// Exchange of the row-sharded path: gathers `count` doubles from every rank into
// `all` (size * count doubles, rank order), ordered on stream st. 0 on success.
typedef int (*ShardGatherFn)(void* ctx, const double* mine, double* all, long long count, cudaStream_t st);

// Row-sharded TSQR of this rank's rows X[0:m_local, c0:c0+nc] (TR-row tiles
// [t0[rank], t0[rank] + nt[rank]) of T). `mine` holds maxt * nc * nc doubles and
// `all` size times that; ws holds tsqr_workspace_doubles(T * TR, nc). R is
// written on every rank.
struct TsqrShard {
    int rank = 0, size = 1;
    i64 T = 0, maxt = 0;
    const i64* t0 = nullptr;   // first tile of each rank
    const i64* nt = nullptr;   // tiles of each rank
    double* mine = nullptr;
    double* all = nullptr;
    ShardGatherFn gather = nullptr;
    void* ctx = nullptr;
};
int launch_tsqr_sharded(double* X, i64 ld, i64 m_local, int c0, int nc, double* R, int ldR, double* ws,
                        const TsqrShard& sh, cudaStream_t st);

// Gram partials only: part[c][i + j*na] = rows [c*rows, (c+1)*rows) of
// X[:, a0:a0+na]^T X[:, b0:b0+nb], for the ceil(m / rows) chunks of exactly
// `rows` rows (a multiple of 32; the last chunk is cut at m). Each chunk is summed
// in segments of 256 rows, so accuracy does not degrade with `rows`.
int launch_gram_partials_fp64(const double* X, i64 ld, i64 m, int a0, int na, int b0, int nb, double* part,
                              i64 rows, cudaStream_t st);

// Accuracy metrics (the reference's test_orth_accuracy, SRC/util.c:36-75).
// E (n x n, lde) = G - I from the upper triangle of the Gram G (ld ldg), mirrored;
// out[0] = ||E||_F (double-double accumulation, fixed order).
int launch_loo_finish(const double* G, int ldg, int n, double* E, int lde, double* out, cudaStream_t st);
// out[1] = ||Q R - X||_F (R upper: entries below its diagonal are not read) and
// out[2] = ||X||_F; part holds metrics_part_doubles(m, n) doubles.
i64 metrics_part_doubles(i64 m, int n);
int launch_residual(const double* X, i64 ldx, const double* Q, i64 ldq, i64 m, int n, const double* R, int ldr,
                    double* part, double* out, cudaStream_t st);

}  // namespace bcgs
