// sytrd_f32.cu — the mixed path's one-stage Householder reduction
// (sytrd_cluster.cuh in FP32).
#include "sytrd_small.cuh"

namespace fkg {

// Several CTAs on an SM overlap each other's barriers but share its shared
// memory among their tiles; measured ms (NB = 4; 4 | 8 | 16 warps): 512 chains of
// N = 144 0.62 | 0.96, 304 of N = 144 0.51 | 0.49, 512 of N = 256 1.62 | 2.18, 304 of
// N = 256 1.30 | 1.10 | 1.82, 304 of N = 400 3.71 | 3.12 | 3.98, 128 of N = 400 - | 2.28 |
// 2.00, 256 of N = 576 - | 8.5 | 7.9, one of N = 1024 - | 7.2 | 6.4. Panels of 8
// instead of 4 read and write tiles in global memory less often, but their rows of V
// and W take the shared memory of 8 tiles at N = 1024 and their corrections twice the
// work: 128 chains of N = 1024 25.7 (8), 25.1 (4); 304 of N = 784 24.6, 23.6; 1024 of N =
// 144 .. 1024 34.9, 32.8.
cudaError_t launch_sytrd_f32(const ChainDesc* h_desc, const ChainDesc* d_desc, int batch, int max_ld,
                             const double* d_diag, float* d_A, void* d_spill, double* d_d, double* d_e, float* d_tau,
                             cudaStream_t st, const int* d_order, int* d_counter, int num_sms, int* d_status) {
    if (batch <= 0) return cudaSuccess;
    if (max_ld <= 128) {
        auto* small = max_ld <= 32   ? launch_small<F32<8>, 32, 8>
                      : max_ld <= 64 ? launch_small<F32<8>, 64, 8>
                      : max_ld <= 96 ? launch_small<F32<8>, 96, 8>
                                     : launch_small<F32<8>, 128, 4>;
        return small(d_desc, batch, d_diag, d_A, d_d, d_e, d_tau, d_order, d_status, st);
    }
    const bool narrow = max_ld <= 256 || (max_ld <= 480 && batch > num_sms);
    auto* launch = max_ld <= 256 && batch > 2 * num_sms ? launch_cluster<F32<4>, 4>
                   : narrow                     ? launch_cluster<F32<8>, 4>
                                                   : launch_cluster<F32<16>, 4>;
    return launch(h_desc, d_desc, batch, max_ld, d_diag, d_A, d_spill, d_d, d_e, d_tau, d_order, d_counter, num_sms,
                  d_status, st);
}

}  // namespace fkg
