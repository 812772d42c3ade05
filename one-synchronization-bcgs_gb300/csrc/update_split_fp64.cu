// Update kernels that split K over a CTA's four warps, and the batched form.
#include "update_fp64.cuh"

namespace bcgs {

int launch_update_split_k(double* X, i64 ld, i64 m, int q0, int K, int c0, int nc, const double* S, int lds,
                          const double* T, int ldt, const int* gate, cudaStream_t st) {
    return launch_update_width<true>(X, ld, m, q0, K, c0, nc, S, lds, T, ldt, gate, st);
}

// ---------------------------------------------------------------------------
// Batched form: one launch over many matrices' jobs (batched.h), each with the single
// launch's split rule and so its arithmetic.
// ---------------------------------------------------------------------------
void update_batched_ctas(i64 m, int K, int* split, int* ctas) {
    *split = up_split(m, K) ? 1 : 0;
    *ctas = (int)ceil_div(m, *split ? 32 : UP_THREADS);
}

__global__ void __launch_bounds__(UP_THREADS)
update_batched(const UpdJob* __restrict__ jobs, const int* __restrict__ prefix, int njobs) {
    __shared__ double sm[up_smem<16, true>() > up_smem<16, false>() ? up_smem<16, true>() : up_smem<16, false>()];
    const int j = batched_job_of(prefix, njobs, blockIdx.x);
    const UpdJob J = jobs[j];
    const i64 blk = blockIdx.x - prefix[j];
#define BCGS_UB(N)                                                                                                \
    if (J.nc <= N) {                                                                                              \
        if (J.split)                                                                                              \
            update_body<N, true>(J.X, J.ld, J.m, J.q0, J.K, J.c0, J.nc, J.S, J.lds, J.T, J.ldt, blk, sm);           \
        else                                                                                                      \
            update_body<N, false>(J.X, J.ld, J.m, J.q0, J.K, J.c0, J.nc, J.S, J.lds, J.T, J.ldt, blk, sm);          \
        return;                                                                                                   \
    }
    BCGS_UB(4) BCGS_UB(8) BCGS_UB(12) BCGS_UB(16)
#undef BCGS_UB
}

int launch_update_batched(const UpdJob* jobs, const int* prefix, int njobs, int items, cudaStream_t st) {
    if (items <= 0) return 0;
    update_batched<<<(unsigned)items, UP_THREADS, 0, st>>>(jobs, prefix, njobs);
    g_launch_count += 1;
    return (int)cudaGetLastError();
}

}  // namespace bcgs
