// sytrd_f64.cu — the FP64 path's Householder reduction (sytrd_cluster.cuh with
// two-limb fixed-point arithmetic).
#include "sytrd_small.cuh"

namespace fkg {

// variant: panel width 2 or 4 (fkg_set_tuning)
cudaError_t launch_sytrd_f64(const ChainDesc* h_desc, const ChainDesc* d_desc, int batch, int max_ld,
                             const double* d_diag, double* d_A, void* d_spill, double* d_d, double* d_e,
                             double* d_tau, cudaStream_t st, int variant, const int* d_order, int* d_counter,
                             int* d_status) {
    if (batch <= 0) return cudaSuccess;
    if (max_ld <= 128) {
        auto* small = max_ld <= 32   ? launch_small<Fix<28>, 32, 8>
                      : max_ld <= 64 ? launch_small<Fix<28>, 64, 8>
                      : max_ld <= 96 ? launch_small<Fix<28>, 96, 8>
                                     : launch_small<Fix<28>, 128, 4>;
        return small(d_desc, batch, d_diag, d_A, d_d, d_e, d_tau, d_order, d_status, st);
    }
    auto* launch = variant == 0 ? launch_cluster<Fix<27>, 2> : launch_cluster<Fix<27>, 4>;
    return launch(h_desc, d_desc, batch, max_ld, d_diag, d_A, d_spill, d_d, d_e, d_tau, d_order, d_counter, d_status,
                  st);
}

}  // namespace fkg
