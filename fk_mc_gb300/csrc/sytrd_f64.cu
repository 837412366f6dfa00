// sytrd_f64.cu — the FP64 path's Householder reduction (sytrd_cluster.cuh with
// two-limb fixed-point arithmetic).
#include "sytrd_small.cuh"

namespace fkg {

// variant: panel width 2 or 4 (fkg_set_tuning)
cudaError_t launch_sytrd_f64(const ChainDesc* h_desc, const ChainDesc* d_desc, int batch, int max_ld,
                             const double* d_diag, double* d_A, void* d_spill, double* d_d, double* d_e,
                             double* d_tau, cudaStream_t st, int variant, const int* d_order, int* d_counter,
                             int num_sms, int* d_status) {
    if (batch <= 0) return cudaSuccess;
    if (max_ld <= 128) {
        auto* small = max_ld <= 32   ? launch_small<Fix<28, 8>, 32, 8>
                      : max_ld <= 64 ? launch_small<Fix<28, 8>, 64, 8>
                      : max_ld <= 96 ? launch_small<Fix<28, 8>, 96, 8>
                                     : launch_small<Fix<28, 8>, 128, 4>;
        return small(d_desc, batch, d_diag, d_A, d_d, d_e, d_tau, d_order, d_status, st);
    }
    // Two CTAs of 4 warps on an SM overlap each other's barriers and scalar phases,
    // at half the shared memory and warps for each; measured ms (4 | 8 warps): 512 chains of
    // N = 144 2.39 | 3.42, N = 256 6.6 | 8.5, N = 324 14.6 | 16.2, N = 400 23.8 | 24.3,
    // N = 576 62 | 60; 152 chains of N = 256 2.39 | 2.14.
    const bool narrow = max_ld <= 384 && batch > num_sms;
    auto* launch = variant == 0 ? (narrow ? launch_cluster<Fix<27, 4>, 2> : launch_cluster<Fix<27, 8>, 2>)
                                : (narrow ? launch_cluster<Fix<27, 4>, 4> : launch_cluster<Fix<27, 8>, 4>);
    return launch(h_desc, d_desc, batch, max_ld, d_diag, d_A, d_spill, d_d, d_e, d_tau, d_order, d_counter, num_sms,
                  d_status, st);
}

}  // namespace fkg
