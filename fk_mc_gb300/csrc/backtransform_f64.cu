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
// A warp holds whole columns of Z in registers (lane: rows lane + 32 r; two columns up to n = 384, one above, where
// two would leave two warps a scheduler) and applies the reflectors in blocks of four, Q_b = I - V T V^T: four dot
// products a column, reduced by shuffles, the 4 x 4 product in 128-bit integers, one update. Four to a block halve
// the rounding of one by one (one rounding per block and entry) and share the shuffles. V is turned into limbs once
// per chain and copied to shared memory one block ahead. Bound by the integer pipes: about 100 cycles a scheduler
// for 32 rows of a column and a block, 17 ms at 256 x N = 576.
// Measured: 32 chains of N = 225 1.87 -> 0.43 ms, 256 of N = 576 126 -> 35 ms, 32 of N = 1024 77 -> 26 ms
// (two columns a warp throughout: 44 and 28).
#include "sytrd_cluster.cuh"

namespace fkg {
namespace {

using FX = Fix<27, 8>;
constexpr int kBlk = 4;        // reflectors to a block
constexpr double kOne = 0x1p57;

__device__ __forceinline__ void cp_async8(void* smem, const void* g, bool ok) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(g),
                 "r"(ok ? 8 : 0)
                 : "memory");
}

// first row of a block's reflectors that the update touches, in units of 32, and of the dot products (pairs of 32)
__device__ __forceinline__ int first_row(int b) { return (b * kBlk + 1) >> 5; }

// One warp per block of four reflectors: their T (quantum 2^-54; its columns are coefficient vectors of at most four
// reflectors, |T| < 2^9) from the dot products, and the reflectors in place as two limbs, unit and zeros included,
// so that the columns' CTAs stage them without a conversion.
// T from its inverse diag(1/tau) + triu(V^T V, 1), as larft_kernel.
__global__ void __launch_bounds__(256)
reflectors_fix_kernel(const ChainDesc* __restrict__ descs, double* __restrict__ Aws, const double* __restrict__ tau,
                      ll* __restrict__ Tf) {
    const ChainDesc D = descs[blockIdx.y];
    const int n = D.n, ld = D.ld, lane = threadIdx.x & 31, b = blockIdx.x * 8 + (threadIdx.x >> 5), k0 = b * kBlk;
    if (k0 >= n - 2) return;
    double* A = Aws + D.a_off + (size_t)k0 * ld;
    FX::Acc acc[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) FX::zero(acc[q]);
    for (int i = (first_row(b) & ~1) * 32 + lane; i < n; i += 32) {
        int2 v[kBlk];
#pragma unroll
        for (int l = 0; l < kBlk; ++l) {
            const int k = k0 + l;
            const double x = k >= n - 2 || i <= k ? 0.0 : i == k + 1 ? 1.0 : A[(size_t)l * ld + i];
            v[l] = FX::split(__double2ll_rn(x * kOne));
            if (k < n - 2) ((int2*)A)[(size_t)l * ld + i] = v[l];
        }
        int q = 0;
#pragma unroll
        for (int l = 0; l < kBlk; ++l)
#pragma unroll
            for (int m = l + 1; m < kBlk; ++m, ++q) FX::mac(acc[q], v[l], v[m]);
    }
    double G[kBlk][kBlk], T[kBlk][kBlk];
    {
        int q = 0;
#pragma unroll
        for (int l = 0; l < kBlk; ++l)
#pragma unroll
            for (int m = l + 1; m < kBlk; ++m, ++q) G[l][m] = (double)warp_sum_ll(FX::sum(acc[q])) * 0x1p-60;
    }
#pragma unroll
    for (int j = 0; j < kBlk; ++j)
#pragma unroll
        for (int r = kBlk - 1; r >= 0; --r) {
            const double tr = k0 + r < n - 2 ? tau[D.v_off + k0 + r] : 0.0;
            double s = 0.0;
#pragma unroll
            for (int q = r + 1; q <= j; ++q) s += G[r][q] * T[q][j];
            T[r][j] = r > j ? 0.0 : r == j ? tr : -tr * s;
        }
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < kBlk * kBlk; ++q) t = lane == q ? T[q / kBlk][q % kBlk] : t;
    if (lane < kBlk * kBlk) Tf[4 * D.v_off + (size_t)b * kBlk * kBlk + lane] = __double2ll_rn(t * 0x1p54);
}

// R rows a lane (n <= 32 R), W warps, NC columns a warp
template <int R, int W, int NC, int OCC>
__global__ void __launch_bounds__(W * 32, OCC)
backtransform_fix_kernel(const ChainDesc* __restrict__ descs, const double* __restrict__ Aws,
                         const ll* __restrict__ Tf, double* __restrict__ Zws) {
    constexpr int kSpan = 32 / (NC * kBlk);  // lanes that hold one reduced sum
    extern __shared__ __align__(16) int2 vs[];  // [2][kBlk / 2][32 R][2]: a lane's 16 bytes hold a pair of reflectors
    const ChainDesc D = descs[blockIdx.y];
    const int n = D.n, ld = D.ld;
    if ((int)blockIdx.x * NC * W >= n) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int2* __restrict__ A = (const int2*)(Aws + D.a_off);
    const ll* __restrict__ T = Tf + 4 * D.v_off;
    double* __restrict__ Z = Zws + D.a_off;
    const int j0 = (blockIdx.x * W + warp) * NC;
    int2 z[NC][R];
    bool bad[NC] = {};  // a NaN stays one: no fixed-point number stands for it
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int i = lane + 32 * r;
            const double x = i < n && j0 + c < n ? Z[(size_t)i * ld + j0 + c] : 0.0;
            bad[c] |= !(fabs(x) < 2.0);
            z[c][r] = FX::split(__double2ll_rn(x * kOne));
        }
#pragma unroll
    for (int c = 0; c < NC; ++c) bad[c] = __any_sync(0xffffffffu, bad[c]);
    const int nblk = n > 2 ? (n - 2 + kBlk - 1) / kBlk : 0;
    auto stage = [&](int b) {
        int2* buf = vs + (size_t)(b & 1) * 32 * R * kBlk;
#pragma unroll
        for (int l = 0; l < kBlk; ++l) {
            const int k = b * kBlk + l;
            for (int i = (first_row(b) & ~1) * 32 + tid; i < 32 * R; i += W * 32) {
                const bool ok = k < n - 2 && i < n;
                cp_async8(buf + ((l >> 1) * 32 * R + i) * 2 + (l & 1), ok ? A + (size_t)k * ld + i : A, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (nblk > 0) stage(nblk - 1);
    for (int b = nblk - 1; b >= 0; --b) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // block b staged; the other buffer's readers are done
        if (b > 0) stage(b - 1);
        ll tl[kBlk];  // T's row of this lane's coefficient (idx below)
#pragma unroll
        for (int l = 0; l < kBlk; ++l) tl[l] = T[(size_t)(b * kBlk + lane / (32 / kBlk)) * kBlk + l];
        const int r0 = first_row(b);  // rows below 32 r0 are zero in V
        const int2* v = vs + (size_t)(b & 1) * 32 * R * kBlk + (size_t)lane * 2;
        if (j0 < n) {
            // W = V^T z
            FX::Acc acc[kBlk][NC];
#pragma unroll
            for (int l = 0; l < kBlk; ++l)
#pragma unroll
                for (int c = 0; c < NC; ++c) FX::zero(acc[l][c]);
#pragma unroll
            for (int r = 0; r < R; r += 2)
                if (r + 1 >= r0) {
#pragma unroll
                    for (int l = 0; l < kBlk; l += 2) {
                        int2 va[2], vb[2];
                        FX::ld2(v + (l * 16 * R + 32 * r) * 2, va);
                        FX::ld2(v + (l * 16 * R + 32 * (r + 1)) * 2, vb);
#pragma unroll
                        for (int h = 0; h < 2; ++h)
#pragma unroll
                            for (int c = 0; c < NC; ++c) FX::mac2(acc[l + h][c], va[h], z[c][r], vb[h], z[c][r + 1]);
                    }
                }
            ll x[NC * kBlk];
#pragma unroll
            for (int l = 0; l < kBlk; ++l)
#pragma unroll
                for (int c = 0; c < NC; ++c) x[NC * l + c] = FX::sum(acc[l][c]);
            int idx;
            ll w = reduce_scatter<NC * kBlk, 16>(x, lane, idx);
#pragma unroll
            for (int o = kSpan / 2; o > 1; o >>= 1) w = add_mod(w, __shfl_xor_sync(0xffffffffu, w, o));
            w = add_mod(w, __shfl_xor_sync(0xffffffffu, w, 1));  // lanes kSpan idx ..: W(idx / NC, column idx % NC), 2^-60
            // W2 = T W, 2^-114 -> quantum 2^-56
            __int128 s = 0;
#pragma unroll
            for (int l = 0; l < kBlk; ++l)
                s += (__int128)tl[l] * __shfl_sync(0xffffffffu, w, (NC * l + idx % NC) * kSpan);
            const int2 w2 = FX::split((ll)((s + ((__int128)1 << 57)) >> 58));
            int2 wv[kBlk][NC];
#pragma unroll
            for (int l = 0; l < kBlk; ++l)
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    wv[l][c] = make_int2(__shfl_sync(0xffffffffu, w2.x, (NC * l + c) * kSpan),
                                         __shfl_sync(0xffffffffu, w2.y, (NC * l + c) * kSpan));
            // z -= V W2 (2^-30 x 2^-29 units, as the reduction's rank-2k update)
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r >= r0) {
                    int2 va[2], vb[2];
                    FX::ld2(v + 32 * r * 2, va);
                    FX::ld2(v + (32 * R + 32 * r) * 2, vb);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        FX::Acc u;
                        FX::zero(u);
                        FX::mac2(u, va[0], wv[0][c], va[1], wv[1][c]);
                        FX::mac2(u, vb[0], wv[2][c], vb[1], wv[3][c]);
                        z[c][r] = FX::upd(z[c][r], u);
                    }
                }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int i = lane + 32 * r;
            if (i < n && j0 + c < n)
                Z[(size_t)i * ld + j0 + c] = bad[c] ? (double)NAN : (double)FX::join(z[c][r]) * (1.0 / kOne);
        }
}

template <int R, int W, int NC, int OCC>
cudaError_t launch_fix(const ChainDesc* d_desc, int batch, int max_n, const double* d_A, const ll* d_Tf,
                       double* d_Z, cudaStream_t st) {
    const size_t smem = sizeof(int2) * 2 * 32 * R * kBlk;
    auto* kern = backtransform_fix_kernel<R, W, NC, OCC>;
    const cudaError_t err = allow_smem<backtransform_fix_kernel<R, W, NC, OCC>>();
    if (err != cudaSuccess) return err;
    kern<<<dim3((max_n + NC * W - 1) / (NC * W), batch), W * 32, smem, st>>>(d_desc, d_A, d_Tf, d_Z);
    return cudaGetLastError();
}

}  // namespace

// X = Q Z with Z row-major in global memory; the reflectors in d_A are turned into fixed point in place (d_Tf: 4
// numbers a row). The instances differ in the rows a lane holds and the columns a warp holds.
cudaError_t launch_backtransform_f64(const ChainDesc* d_desc, int batch, int max_n, double* d_A, const double* d_tau,
                                     long long* d_Tf, double* d_Z, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    if (batch > 65535) return cudaErrorInvalidValue;  // grid y limit
    reflectors_fix_kernel<<<dim3((max_n + 8 * kBlk - 1) / (8 * kBlk), batch), 256, 0, st>>>(d_desc, d_A, d_tau, d_Tf);
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    auto* launch = max_n <= 64    ? launch_fix<2, 8, 2, 2>
                   : max_n <= 128 ? launch_fix<4, 8, 2, 2>
                   : max_n <= 256 ? launch_fix<8, 8, 2, 2>
                   : max_n <= 384 ? launch_fix<12, 8, 2, 2>
                   : max_n <= 576 ? launch_fix<18, 8, 1, 2>
                   : max_n <= 768 ? launch_fix<24, 8, 1, 2>
                                  : launch_fix<32, 8, 1, 2>;
    return launch(d_desc, batch, max_n, d_A, d_Tf, d_Z, st);
}

}  // namespace fkg
