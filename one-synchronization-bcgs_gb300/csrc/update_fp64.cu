// Update kernels with the whole K per row, and the choice between them and the split form.
#include "update_fp64.cuh"

namespace bcgs {

int launch_update_fp64(double* X, i64 ld, i64 m, int q0, int K, int c0, int nc, const double* S, int lds,
                       const double* T, int ldt, bool any_split, cudaStream_t st, const int* gate) {
    if (nc <= 0 || m <= 0) return 0;
    if (any_split && up_split(m, K) && nc <= 32)
        return launch_update_split_k(X, ld, m, q0, K, c0, nc, S, lds, T, ldt, gate, st);
    return launch_update_width<false>(X, ld, m, q0, K, c0, nc, S, lds, T, ldt, gate, st);
}

}  // namespace bcgs
