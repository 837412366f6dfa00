// backtransform_f64.cu — X = Q Z of the FP64 path (calc_ed(true),
// src/configuration.cpp:216-219): the reduction's reflectors applied to the
// tridiagonal's eigenvectors.
//
// A contraction of n^3 multiply-adds that GB300's FP64 pipe makes at one per
// warp in 64-76 cycles; here, as in the reduction (sytrd_cluster.cuh, struct
// Fix), entries are two-limb fixed-point numbers and a product is three
// integer multiplications. Eigenvectors and reflectors are bounded by 1 (quantum
// 2^-57), the dot products by sqrt(2), the coefficients T V^T z by 2: they are
// tau_l v_l . (H_{l+1} .. H_4 z) with |z| = 1 and tau |v| = 2 / |v| <= 2.
//
// A warp holds two whole columns of Z in registers (lane: rows lane + 32 r) and
// applies the reflectors in blocks of four, Q_b = I - V T V^T with T the 4 x 4
// diagonal block of larft's panel factor: four dot products a column, reduced
// by shuffles, the 4 x 4 product in 128-bit integers, one update. Four to a
// block halve the rounding of one by one (one rounding per block and entry) and share the
// shuffles. The CTA's warps share V, staged as integers one block ahead.
// Measured: 32 chains of N = 225 1.87 -> 0.73 ms, 256 of N = 576 126 -> 62 ms.
#include "sytrd_cluster.cuh"

namespace fkg {
namespace {

using FX = Fix<27, 8>;
constexpr int kBlk = 4;        // reflectors to a block
constexpr int kPanel = 32;     // larft's panel
constexpr double kOne = 0x1p57;

// R rows a lane (n <= 32 R), W warps, two columns a warp
template <int R, int W>
__global__ void __launch_bounds__(W * 32)
backtransform_fix_kernel(const ChainDesc* __restrict__ descs, const double* __restrict__ Aws,
                         const double* __restrict__ Tf, double* __restrict__ Zws) {
    constexpr int kThreads = W * 32, kPf = kBlk * R / W;  // entries of V staged a thread and block
    static_assert(kBlk * R % W == 0, "whole entries a thread");
    extern __shared__ __align__(16) int2 vs[];  // [2][32 R][kBlk]
    __shared__ ll ts[2][kBlk][kBlk];
    const ChainDesc D = descs[blockIdx.y];
    const int n = D.n, ld = D.ld;
    if ((int)blockIdx.x * 2 * W >= n) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double* __restrict__ A = Aws + D.a_off;
    const double* __restrict__ T = Tf + (D.v_off / kPanel) * (size_t)(kPanel * kPanel);
    double* __restrict__ Z = Zws + D.a_off;
    const int j0 = (blockIdx.x * W + warp) * 2;
    int2 z[2][R];
    bool bad[2] = {false, false};  // a NaN stays one: no fixed-point number stands for it
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int i = lane + 32 * r;
            const double x = i < n && j0 + c < n ? Z[(size_t)i * ld + j0 + c] : 0.0;
            bad[c] |= !(fabs(x) < 2.0);
            z[c][r] = FX::split(__double2ll_rn(x * kOne));
        }
#pragma unroll
    for (int c = 0; c < 2; ++c) bad[c] = __any_sync(0xffffffffu, bad[c]);
    const int nblk = n > 2 ? (n - 2 + kBlk - 1) / kBlk : 0;
    // entry e of a block: reflector e / (32 R), row e % (32 R)
    double pf[kPf], pt = 0.0;
    auto fetch = [&](int b) {
#pragma unroll
        for (int q = 0; q < kPf; ++q) {
            const int e = tid + kThreads * q, k = b * kBlk + e / (32 * R), i = e % (32 * R);
            double v = 0.0;
            if (k < n - 2 && i < n) {
                if (i == k + 1) v = 1.0;
                else if (i > k + 1) v = A[(size_t)k * ld + i];
            }
            pf[q] = v;
        }
        if (tid < kBlk * kBlk) {
            const int k = b * kBlk, o = k % kPanel;
            pt = T[(size_t)(k / kPanel) * kPanel * kPanel + (o + tid / kBlk) * kPanel + o + tid % kBlk];
        }
    };
    auto stage = [&](int buf) {
#pragma unroll
        for (int q = 0; q < kPf; ++q) {
            const int e = tid + kThreads * q;
            vs[(size_t)buf * 32 * R * kBlk + (e % (32 * R)) * kBlk + e / (32 * R)] =
                FX::split(__double2ll_rn(pf[q] * kOne));
        }
        // |T| < 2^9: its columns are coefficient vectors of at most four reflectors
        if (tid < kBlk * kBlk) ts[buf][tid / kBlk][tid % kBlk] = __double2ll_rn(pt * 0x1p54);
    };
    if (nblk > 0) {
        fetch(nblk - 1);
        stage((nblk - 1) & 1);
    }
    for (int b = nblk - 1; b >= 0; --b) {
        __syncthreads();  // block b staged; the other buffer's readers are done
        if (b > 0) fetch(b - 1);
        const int buf = b & 1, r0 = (b * kBlk + 1) >> 5;  // rows below 32 r0 are zero in V
        const int2* v = vs + (size_t)buf * 32 * R * kBlk + (size_t)lane * kBlk;
        if (j0 < n) {
            // W = V^T z
            FX::Acc acc[kBlk][2];
#pragma unroll
            for (int l = 0; l < kBlk; ++l) {
                FX::zero(acc[l][0]);
                FX::zero(acc[l][1]);
            }
#pragma unroll
            for (int r = 0; r < R; r += 2)
                if (r + 1 >= r0) {
#pragma unroll
                    for (int l = 0; l < kBlk; l += 2) {
                        int2 va[2], vb[2];
                        FX::ld2(v + (size_t)32 * r * kBlk + l, va);
                        FX::ld2(v + (size_t)32 * (r + 1) * kBlk + l, vb);
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int c = 0; c < 2; ++c) FX::mac2(acc[l + h][c], va[h], z[c][r], vb[h], z[c][r + 1]);
                    }
                }
            ll x[2 * kBlk];
#pragma unroll
            for (int l = 0; l < kBlk; ++l) {
                x[2 * l] = FX::sum(acc[l][0]);
                x[2 * l + 1] = FX::sum(acc[l][1]);
            }
            int idx;
            ll w = reduce_scatter<2 * kBlk, 16>(x, lane, idx);
            w = add_mod(w, __shfl_xor_sync(0xffffffffu, w, 2));
            w = add_mod(w, __shfl_xor_sync(0xffffffffu, w, 1));  // lanes 4 idx ..: W(idx / 2, column idx % 2), 2^-60
            // W2 = T W, 2^-114 -> quantum 2^-56
            __int128 s = 0;
#pragma unroll
            for (int l = 0; l < kBlk; ++l)
                s += (__int128)ts[buf][idx >> 1][l] * __shfl_sync(0xffffffffu, w, (2 * l + (idx & 1)) * 4);
            const int2 w2 = FX::split((ll)((s + ((__int128)1 << 57)) >> 58));
            int2 wv[kBlk][2];
#pragma unroll
            for (int l = 0; l < kBlk; ++l)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    wv[l][c] = make_int2(__shfl_sync(0xffffffffu, w2.x, (2 * l + c) * 4),
                                         __shfl_sync(0xffffffffu, w2.y, (2 * l + c) * 4));
            // z -= V W2 (2^-30 x 2^-29 units, as the reduction's rank-2k update)
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r >= r0) {
                    int2 va[2], vb[2];
                    FX::ld2(v + (size_t)32 * r * kBlk, va);
                    FX::ld2(v + (size_t)32 * r * kBlk + 2, vb);
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        FX::Acc u;
                        FX::zero(u);
                        FX::mac2(u, va[0], wv[0][c], va[1], wv[1][c]);
                        FX::mac2(u, vb[0], wv[2][c], vb[1], wv[3][c]);
                        z[c][r] = FX::upd(z[c][r], u);
                    }
                }
        }
        if (b > 0) stage((b - 1) & 1);
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int i = lane + 32 * r;
            if (i < n && j0 + c < n)
                Z[(size_t)i * ld + j0 + c] = bad[c] ? (double)NAN : (double)FX::join(z[c][r]) * (1.0 / kOne);
        }
}

template <int R, int W>
cudaError_t launch_fix(const ChainDesc* d_desc, int batch, int max_n, const double* d_A, const double* d_Tf,
                       double* d_Z, cudaStream_t st) {
    const size_t smem = sizeof(int2) * 2 * 32 * R * kBlk;
    auto* kern = backtransform_fix_kernel<R, W>;
    const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    kern<<<dim3((max_n + 2 * W - 1) / (2 * W), batch), W * 32, smem, st>>>(d_desc, d_A, d_Tf, d_Z);
    return cudaGetLastError();
}

}  // namespace

// d_Tf: the panels' factors (larft_kernel); the instances differ in the rows a lane holds
cudaError_t launch_backtransform_fix(const ChainDesc* d_desc, int batch, int max_n, const double* d_A,
                                     const double* d_Tf, double* d_Z, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    if (batch > 65535) return cudaErrorInvalidValue;  // grid y limit
    auto* launch = max_n <= 64    ? launch_fix<2, 8>
                   : max_n <= 128 ? launch_fix<4, 8>
                   : max_n <= 256 ? launch_fix<8, 8>
                   : max_n <= 384 ? launch_fix<12, 8>
                   : max_n <= 576 ? launch_fix<18, 8>
                   : max_n <= 768 ? launch_fix<24, 8>
                                  : launch_fix<32, 8>;
    return launch(d_desc, batch, max_n, d_A, d_Tf, d_Z, st);
}

}  // namespace fkg
