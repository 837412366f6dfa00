// sytrd_small.cuh — Householder tridiagonalisation of orders up to 128, one CTA
// per chain with the whole symmetric matrix in registers.
//
// The same mathematics and arithmetic (template parameter P: F32 or Fix) as
// sytrd_cluster.cuh, laid out for latency, which is all that bounds these
// orders: a column of the tiled kernel costs ~9 k cycles at N = 64 whatever the
// work in it. Thread (r, q) owns row r and the columns c = q mod G, both triangles
// stored; a warp holds 32 / G whole rows, so a matrix-vector product ends with
// log2 G shuffles, needs no column sums, and the rank-2 update follows at once
// (no panels, no corrections). One warp forms the reflector from the column
// (= the row that its owner wrote after the last update); four barriers a
// column. Rows and columns that are done are skipped. Measured per solve (ms;
// tiled kernel, this one): FP64 arithmetic N = 64 0.28, 0.152; 512 chains of N = 64
// 1.08, 0.39; N = 121 0.68, 0.54; FP32 N = 64 0.158, 0.068; 512 chains 0.34, 0.142;
// N = 121 0.34, 0.18.
#pragma once
#include "sytrd_cluster.cuh"

namespace fkg {
namespace {

template <class P, int R, int G>
struct SmallSmem {
    static constexpr int E = R / G, kStride = E + 2;  // padded: conflict-free reads of G column groups
    typename P::V vq[G * kStride], wq[G * kStride];   // v and w by column group
    typename P::S x[R];                               // column k
    typename P::S pvp[R * G / 32];
    typename P::S dr[R], er[R];
    ull tr[R];
    double rs[R], red[R * G / 32];
    FixRefl refl;
    float tau, beta, scale;
    typename P::V mat[R * (R + 1)];  // the matrix while it is built (last: see small_smem)
};

template <class P, int R, int G>
__global__ void __launch_bounds__(R * G)
sytrd_small_kernel(const ChainDesc* __restrict__ descs, const double* __restrict__ diag,
                   typename P::G* __restrict__ Aout, double* __restrict__ dout, double* __restrict__ eout,
                   typename P::G* __restrict__ tauout, const int* __restrict__ order, int* __restrict__ status) {
    using V = typename P::V;
    using S = typename P::S;
    using Acc = typename P::Acc;
    constexpr bool kFix = sizeof(S) == 8;
    constexpr int E = R / G, kThreads = R * G, kWarps = kThreads / 32, kStride = E + 2;
    extern __shared__ __align__(16) unsigned char sm_raw[];
    auto& M = *reinterpret_cast<SmallSmem<P, R, G>*>(sm_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = tid % G, r = tid / G;
    const ChainDesc D = descs[order ? order[blockIdx.x] : blockIdx.x];
    const int n = D.n, ld = D.ld;
    typename P::G* __restrict__ A = Aout + D.a_off;
    const int rowslot = (r % G) * kStride + r / G;  // row r as a column index

    // ---- build in shared memory (entries j <= i, mirrored), then to registers ----
    for (int i = tid; i < R * (R + 1); i += kThreads) M.mat[i] = P::vzero();
    for (int i = tid; i < G * kStride; i += kThreads) M.vq[i] = M.wq[i] = P::vzero();
    double quant = 1.0, inv = 1.0;
    if constexpr (kFix) {
        for (int i = tid; i < R; i += kThreads) M.rs[i] = 0.0;
        __syncthreads();
        for (int i = tid; i < n; i += kThreads) {
            double own = fabs(diag[D.v_off + i]);
#pragma unroll 1
            for (int p = D.rowptr[i]; p < D.rowptr[i + 1]; ++p) {
                const int j = D.col[p];
                if ((unsigned)j > (unsigned)i) continue;
                const double a = fabs(D.val[p]);
                own += a;
                if (j < i) atomicAdd(&M.rs[j], a);
            }
            atomicAdd(&M.rs[i], own);
        }
        __syncthreads();
        double m = 0.0;
        bool bad = false;
        for (int i = tid; i < n; i += kThreads) {
            m = fmax(m, M.rs[i]);
            bad = bad || !(M.rs[i] < 0x1p900);
        }
        m = block_max(m, M.red);
        if (__syncthreads_or(bad)) {  // NaN, Inf or out of the format's range
            if (tid == 0 && status) atomicOr(status, kStatusNaN);
            for (int i = tid; i < n; i += kThreads) {
                dout[D.v_off + i] = NAN;  // and so every eigenvalue and logZ
                eout[D.v_off + i] = 0.0;
                tauout[D.v_off + i] = 0;
            }
            return;
        }
        const int eS = m > 0x1p-900 ? ilogb(m * (1.0 + 0x1p-30)) + 1 : -899;
        quant = scalbn(1.0, eS - 30 - P::kLo);
        inv = scalbn(1.0, 30 + P::kLo - eS);
    }
    __syncthreads();
    auto add_elem = [&](int i, int j, double a) {
#pragma unroll 1
        for (int side = 0; side < (i == j ? 1 : 2); ++side) {
            V& m = M.mat[side ? j * (R + 1) + i : i * (R + 1) + j];
            if constexpr (kFix) m = P::split(P::join(m) + __double2ll_rn(a * inv));
            else m += (float)a;
        }
    };
    for (int i = tid; i < n; i += kThreads) {
#pragma unroll 1
        for (int p = D.rowptr[i]; p < D.rowptr[i + 1]; ++p) {
            const int j = D.col[p];
            if ((unsigned)j >= (unsigned)n) {  // a column outside [0, n): skipped, the call fails
                if (status) atomicOr(status, kStatusBadArg);
                continue;
            }
            if (j <= i) add_elem(i, j, D.val[p]);
        }
        add_elem(i, i, diag[D.v_off + i]);
    }
    __syncthreads();
    V a[E];
#pragma unroll
    for (int e = 0; e < E; ++e) a[e] = M.mat[r * (R + 1) + e * G + q];
    auto row_to_x = [&]() {  // the owner of a row publishes it as the next column
#pragma unroll
        for (int e = 0; e < E; ++e) {
            if constexpr (kFix) M.x[e * G + q] = P::join(a[e]);
            else M.x[e * G + q] = a[e];
        }
    };
    if (r == 0) row_to_x();
    __syncthreads();

    for (int k = 0; k < n - 2; ++k) {
        const int s = k + 1;
        // ---- (1) reflector by one warp ----
        if (warp == 0) {
            S xi[R / 32];
#pragma unroll
            for (int m = 0; m < R / 32; ++m) {
                const int i = lane + 32 * m;
                xi[m] = i >= s && i < n ? M.x[i] : S(0);
            }
            const S alpha = M.x[s];
            bool flat;
            float scale = 0.f, tau = 0.f, beta = 0.f;
            FixRefl Rf;
            if constexpr (kFix) {
                ll hh = 0, hl = 0, l2 = 0;
#pragma unroll
                for (int m = 0; m < R / 32; ++m) {
                    const V xv = P::split(xi[m]);
                    hh += (ll)xv.x * xv.x;
                    hl += (ll)xv.x * xv.y;
                    l2 += (ll)xv.y * xv.y;
                }
                hh = warp_sum_ll(hh);
                hl = warp_sum_ll(hl);
                l2 = warp_sum_ll(l2);
                const unsigned __int128 s2 = ((unsigned __int128)(ull)hh << (2 * P::kLo)) +
                                             (unsigned __int128)((__int128)hl << (P::kLo + 1)) + (ull)l2;
                Rf = fix_reflector(s2, alpha);
                flat = Rf.zero;
                if (lane == 0) {
                    M.refl = Rf;
                    const int sh = Rf.z / 2 - 34 + P::kLo;  // 2^-62 S: sqrt(s2) has at most 62 bits there
                    const ll xn = (ll)(sh >= 0 ? Rf.xn >> sh : Rf.xn << -sh);
                    M.er[k] = flat ? alpha << (32 - P::kLo) : (alpha >= 0 ? -xn : xn);
                    M.dr[k] = M.x[k];
                    M.tr[k] = Rf.tau;
                }
            } else {
                float part = 0.f;
#pragma unroll
                for (int m = 0; m < R / 32; ++m) part += lane + 32 * m > s ? xi[m] * xi[m] : 0.f;
                const float sigma = warp_sum(part);
                flat = sigma == 0.f;
                beta = alpha;
                if (!flat) {
                    const float xnorm = sqrtf(alpha * alpha + sigma);
                    beta = alpha >= 0.f ? -xnorm : xnorm;
                    tau = (beta - alpha) / beta;
                    scale = 1.f / (alpha - beta);
                }
                if (lane == 0) {
                    M.tau = tau;
                    M.refl.zero = flat;
                    M.er[k] = beta;
                    M.dr[k] = M.x[k];
                    *(float*)&M.tr[k] = tau;
                }
            }
#pragma unroll
            for (int m = 0; m < R / 32; ++m) {
                const int i = lane + 32 * m;
                V vi = P::vzero();
                if (!flat && i >= s && i < n) {
                    if constexpr (kFix) {
                        ll v = 1ll << (30 + P::kLo);
                        if (i > s) {
                            v = P::template round_to<61, 30 + P::kLo>(__mul64hi(xi[m] << (Rf.z / 2 - 1), (ll)Rf.r));
                            if (alpha < 0) v = -v;
                        }
                        vi = P::split(v);
                    } else {
                        vi = i == s ? 1.f : xi[m] * scale;
                    }
                }
                M.vq[(i % G) * kStride + i / G] = vi;
                if (i > s && i < n) {
                    if constexpr (kFix) {
                        if (Aout) A[(size_t)k * ld + i] = (double)P::join(vi) * (1.0 / (1ll << (30 + P::kLo)));
                    } else {
                        A[(size_t)k * ld + i] = vi;
                    }
                }
            }
        }
        __syncthreads();
        if (M.refl.zero) {  // nothing to apply: publish the next row
            if (r == s) row_to_x();
            __syncthreads();
            continue;
        }
        // ---- (2) p = A v ----
        const bool live = (warp + 1) * (32 / G) > s && warp * (32 / G) < n;  // a row of this warp is left
        const int e0 = s / G;  // column groups below are done
        const V vr = M.vq[rowslot];
        S p = 0;
        if (live) {
            Acc u;
            P::zero(u);
#pragma unroll
            for (int e = 0; e < E; e += 2)
                if (e + 1 >= e0) {
                    V v2[2];
                    P::ld2(M.vq + q * kStride + e, v2);
                    P::mac2(u, a[e], v2[0], a[e + 1], v2[1]);
                }
            p = P::sum(u);
#pragma unroll
            for (int o = G / 2; o >= 1; o >>= 1) p = add_mod(p, __shfl_xor_sync(0xffffffffu, p, o));
            Acc pv;
            P::zero(pv);
            if (q == 0) {
                if constexpr (kFix) P::mac(pv, P::split(P::template round_to<60, 30 + P::kLo>(p)), vr);
                else P::mac(pv, p, vr);
            }
            S pvs = P::sum(pv);
            if constexpr (kFix) pvs = warp_sum_ll(pvs);
            else pvs = warp_sum(pvs);
            if (lane == 0) M.pvp[warp] = pvs;
        } else if (lane == 0) {
            M.pvp[warp] = 0;
        }
        __syncthreads();
        // ---- (3) w = tau p - (tau/2)(tau p . v) v ----
        V wr = P::vzero();
        if (live) {
            S pv = lane < kWarps ? M.pvp[lane] : S(0);
            if constexpr (kFix) {
                pv = warp_sum_ll(pv);
                const ll tau = (ll)M.refl.tau;
                Acc kv;
                P::zero(kv);
                P::mac(kv, P::k_value(pv, tau), vr);
                wr = P::w_entry(p, tau, kv);
            } else {
                pv = warp_sum(pv);
                const float tau = M.tau;
                wr = tau * p - 0.5f * tau * (tau * pv) * vr;
            }
            if (r < s || r >= n) wr = P::vzero();
            if (q == 0) M.wq[rowslot] = wr;
        }
        __syncthreads();
        // ---- (4) A -= v w^T + w v^T ----
        if (live) {
#pragma unroll
            for (int e = 0; e < E; e += 2)
                if (e + 1 >= e0) {
                    V v2[2], w2[2];
                    P::ld2(M.vq + q * kStride + e, v2);
                    P::ld2(M.wq + q * kStride + e, w2);
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        Acc u;
                        P::zero(u);
                        P::mac2(u, vr, w2[b], wr, v2[b]);
                        a[e + b] = P::upd(a[e + b], u);
                    }
                }
            if (r == s) row_to_x();
        }
        __syncthreads();
    }
    // ---- the trailing 2 x 2 block (n <= 2: the whole matrix), then the outputs ----
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int c = e * G + q;
        if (r >= n || r < n - 2 || c < n - 2 || c > r) continue;
        S x;
        if constexpr (kFix) x = P::join(a[e]);
        else x = a[e];
        if (c == r) M.dr[r] = x;
        else if constexpr (kFix) M.er[c] = x << (32 - P::kLo);
        else M.er[c] = x;
    }
    __syncthreads();
    for (int i = tid; i < n; i += kThreads) {
        double* d = dout + D.v_off + i;
        double* e = eout + D.v_off + i;
        if constexpr (kFix) {
            *d = (double)M.dr[i] * quant;
            if (i < n - 1) *e = (double)M.er[i] * (quant / (1ll << (32 - P::kLo)));
            if (Aout && i < n - 2) tauout[D.v_off + i] = (double)M.tr[i] * 0x1p-62;
        } else {
            *d = (double)M.dr[i];
            if (i < n - 1) *e = (double)M.er[i];
            if (i < n - 2) tauout[D.v_off + i] = *(float*)&M.tr[i];
        }
        if (i == n - 2) tauout[D.v_off + i] = 0;
    }
}

}  // namespace

template <class P, int R, int G>
static cudaError_t launch_small(const ChainDesc* d_desc, int batch, const double* d_diag, typename P::G* d_A,
                                double* d_d, double* d_e, typename P::G* d_tau, const int* d_order, int* d_status,
                                cudaStream_t st) {
    auto* kern = sytrd_small_kernel<P, R, G>;
    const int smem = (int)sizeof(SmallSmem<P, R, G>);
    const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (err != cudaSuccess) return err;
    kern<<<batch, R * G, smem, st>>>(d_desc, d_diag, d_A, d_d, d_e, d_tau, d_order, d_status);
    return cudaGetLastError();
}

}  // namespace fkg
