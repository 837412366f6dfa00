// chebyshev.cu — the Chebyshev-expansion logZ of the reference's large-N
// method, configuration_t::calc_chebyshev (src/configuration.cpp:94-205) with
// the coefficients of chebyshev::chebyshev_eval
// (include/fk_mc/chebyshev.hpp:16-66), for a batch of chains:
//
//   1. spectral bounds e_min, e_max of H (the reference asks ARPACK for the
//      smallest and largest eigenvalue): Lanczos on the sparse H, one CTA per
//      chain, in double-float, until the extreme Ritz values stop moving;
//   2. the exact moments mu_m = Tr T_m(x) / N of x = (H - b) / a,
//      a = (e_max - e_min)/2, b = (e_max + e_min)/2, for m < M: the reference
//      forms the matrices T_m(x) for m <= M/2 by the three-term recursion and
//      the rest from Tr(T_{m-1} T_m) and Tr(T_m^2). Here every column j of
//      T_m(x) is built on its own by one warp, T_m(x) e_j = 2 x T_{m-1}(x) e_j
//      - T_{m-2}(x) e_j. That column vanishes outside the sites within m hops
//      of j, so the warp works on the ball of radius M/2 around j only (sites
//      in hop order, the ball's own CSR), in shared memory, in double-float
//      (FP32 pairs: GB300's FP32 pipe is ~60x its FP64 pipe); it adds its
//      column's diagonal entry to Tr T_m and its dot products to Tr(T_{m-1}T_m)
//      and Tr(T_m^2);
//   3. per chain: the column sums in a fixed order, the moments assembled in
//      the reference's order, the coefficients c_m = moment_f(logz_f, m) by the
//      trapezoid rule on the Lobatto grid, logZ = c_0 + sum_m 2 c_m mu_m.
// The Lanczos vectors and the column recursion are double-float (FP32 pairs,
// ~48 bits), the final step FP64; every reduction has a fixed order.
#include "fkg_common.cuh"

namespace fkg {
namespace {

constexpr int kKpmThreads = 256;

// Eigenvalues of the k x k tridiagonal (al, b2 = squared off-diagonal, as
// FP32 pairs) below x, by a pair of lanes from both ends: the even lane takes
// the leading principal minors of the rows above m = k/2, p_0 = 1,
// p_{i+1} = (al_i - x) p_i - b2_{i-1} p_{i-1}, the odd lane those of the rows
// below it from the last one up (q). Their sign changes count the negative
// pivots of the twisted LDL^T factorisation of T - x (Sylvester's inertia); the
// twist's pivot is al_m - x - b2_{m-1} p_{m-1}/p_m - b2_m q'/q, its sign formed from
// the products. Double-float; the minors are rescaled by a common power of two
// when they leave [2^-60, 2^60]; an exact zero counts as a tiny pivot of the
// opposite sign. No division, no FP64 (GB300's FP64 pipe is ~60x narrower than
// FP32), and half the dependent steps of a count from one end (about 150 cycles
// each).
__device__ __forceinline__ int sturm_count(const dfl* al, const dfl* b2, int k, dfl x) {
    const int m = k >> 1;
    const bool odd = threadIdx.x & 1;
    const int len = odd ? k - 1 - m : m;
    const dfl nx = {-x.hi, -x.lo};
    dfl pm = {0.0f, 0.0f}, p = {1.0f, 0.0f};  // the minor before, the minor
    int cnt = 0;
    for (int t = 0; t < m; ++t)
        if (t < len) {
            const int i = odd ? k - 1 - t : t, c = odd ? i : i - 1;  // row, coupling to the row before
            const dfl u = df_mul(df_add(al[i], nx), p);
            dfl q = u;
            if (t > 0) {
                const dfl v = df_mul(b2[c], pm);
                q = df_add(u, {-v.hi, -v.lo});
            }
            if (q.hi == 0.0f) q = {p.hi > 0.0f ? -1e-30f * fabsf(p.hi) : 1e-30f * fabsf(p.hi), 0.0f};
            cnt += (q.hi < 0.0f) != (p.hi < 0.0f);
            pm = p;
            p = q;
            const float ap = fabsf(p.hi);
            if (ap > 0x1p60f || ap < 0x1p-60f) {
                const float sc = ap > 0x1p60f ? 0x1p-60f : 0x1p60f;
                p = {p.hi * sc, p.lo * sc};
                pm = {pm.hi * sc, pm.lo * sc};
            }
        }
    // larger of the two into [1, 2): the products below stay in range
    const float sc = __int_as_float(0x7f000000 - (__float_as_int(fmaxf(fabsf(p.hi), fabsf(pm.hi))) & 0x7f800000));
    p = {p.hi * sc, p.lo * sc};
    pm = {pm.hi * sc, pm.lo * sc};
    const dfl o = {__shfl_xor_sync(0xffffffffu, p.hi, 1), __shfl_xor_sync(0xffffffffu, p.lo, 1)};
    const dfl om = {__shfl_xor_sync(0xffffffffu, pm.hi, 1), __shfl_xor_sync(0xffffffffu, pm.lo, 1)};
    cnt += __shfl_xor_sync(0xffffffffu, cnt, 1);
    const dfl P = odd ? o : p, Pm = odd ? om : pm, Q = odd ? p : o, Qm = odd ? pm : om;
    dfl g = df_mul(df_add(al[m], nx), df_mul(P, Q));
    if (m > 0) {
        const dfl v = df_mul(b2[m - 1], df_mul(Pm, Q));
        g = df_add(g, {-v.hi, -v.lo});
    }
    if (m + 1 < k) {
        const dfl v = df_mul(b2[m], df_mul(Qm, P));
        g = df_add(g, {-v.hi, -v.lo});
    }
    return cnt + (((g.hi < 0.0f) != (P.hi < 0.0f)) != (Q.hi < 0.0f));
}

constexpr int kRitzThreads = 64;               // threads per end of the spectrum
constexpr int kPoints = kRitzThreads / 2;      // a pair of lanes per point

// The first of the group's points (pair order) whose count reaches `want`, kPoints if none does. `slot`
// alternates between calls, so that the next one may write while a slow warp still reads.
__device__ __forceinline__ int first_point(bool reached, int group, int (*slot)[kRitzThreads / 32]) {
    const unsigned mask = __ballot_sync(0xffffffffu, reached);
    const int wid = (threadIdx.x & (kRitzThreads - 1)) >> 5;
    if ((threadIdx.x & 31) == 0) (*slot)[wid] = mask ? wid * 16 + (__ffs(mask) - 1) / 2 : kPoints;
    if (group) asm volatile("bar.sync 2, %0;" ::"n"(kRitzThreads) : "memory");
    else asm volatile("bar.sync 1, %0;" ::"n"(kRitzThreads) : "memory");
    int t = kPoints;
#pragma unroll
    for (int q = 0; q < kRitzThreads / 32; ++q) t = min(t, (*slot)[q]);
    return t;
}

// Smallest (group 0) or largest (group 1) eigenvalue of the tridiagonal by
// multisection, 64 threads per end: a round counts at 32 points, a pair of lanes each.
// It starts from a narrow bracket around the previous Ritz value, whose ends (31/33 span
// away) are two of the first round's points and must hold the eigenvalue,
// else from the Gershgorin bracket, and goes on until the bracket is as narrow
// as the double-float counts resolve (4e-14 relative). Every round cuts into 33rds, the
// first one too: with 31sts it ended at wider brackets (triangular L = 9, U = 0.5: mean error of
// the bounds 2.1e-15, now 1.2e-15).
// One warp per end with counts from one side took 57 % of the bounds kernel.
__device__ double ritz_extreme(const dfl* al, const dfl* b2, int k, double lo, double hi, double prev, double span,
                               bool have_prev, int group, int (*slots)[kRitzThreads / 32]) {
    const int point = (threadIdx.x & (kRitzThreads - 1)) >> 1, want = group ? k : 1;
    int phase = 0;
    if (have_prev) {
        const double step = 2.0 * span * (1.0 / (kPoints + 1)), a = prev - 0.5 * (kPoints - 1) * step;
        const int t = first_point(sturm_count(al, b2, k, df_of(a + step * point)) >= want, group, slots);
        phase = 1;
        if (t > 0 && t < kPoints) {
            lo = a + step * (t - 1);
            hi = a + step * t;
        }
    }
    for (int round = 0; round < 40; ++round) {
        const double w = hi - lo, step = w * (1.0 / (kPoints + 1));
        if (!(w > 4e-14 * fmax(fabs(lo), fabs(hi)))) break;
        const int t = first_point(sturm_count(al, b2, k, df_of(lo + step * (point + 1))) >= want, group, slots + phase);
        phase ^= 1;
        if (t < kPoints) hi = lo + step * (t + 1);
        lo += step * t;
    }
    return 0.5 * (lo + hi);
}

// Block-wide double-float sum, to every thread: each warp's sum through shared
// memory, the cross-warp sum by every thread itself (fixed order), one barrier.
// `red` alternates between two sets of blockDim/32 slots (phase), so that the
// next call may write while a slow warp still reads this one's.
__device__ __forceinline__ dfl block_sum_df(dfl x, float2 (*red)[kKpmThreads / 32], int& phase) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    float2* r = red[phase];
    phase ^= 1;
    x = warp_sum_df(x);
    if (lane == 0) r[wid] = make_float2(x.hi, x.lo);
    __syncthreads();
    dfl t = {0.0f, 0.0f};
    if (lane < nw) t = {r[lane].x, r[lane].y};
    return warp_sum_df(t);
}

// Block-wide (minimum of lo, maximum of hi), to every thread; the caller's next barrier frees `red`
__device__ __forceinline__ float2 block_range(float lo, float hi, float2* red) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (pass) break;
        if (lane == 0) red[threadIdx.x >> 5] = make_float2(lo, hi);
        __syncthreads();
        if (lane < nw) {
            lo = red[lane].x;
            hi = red[lane].y;
        }
    }
    return make_float2(lo, hi);
}

// The Lanczos scalars' square root and reciprocal, to the pair's rounding (2^-49; worst
// 1.8e-15, as a rounded FP64 result): an FP32 estimate, one Newton step, and a
// second one whose residual is formed from error-free products and sums. With one
// step (1e-14 worst) the end of an exhausted Krylov space went unnoticed; a reciprocal of
// the rounded root (2.6e-15) took the bounds' mean error for cubic2d L = 8, U = 0.5 from 2.4e-15 to 7.2e-15.
__device__ __forceinline__ void two_sum32(float a, float b, float& s, float& e) {
    s = a + b;
    const float v = s - a;
    e = (a - (s - v)) + (b - v);
}
// a - b - c - d for a close to b + c + d, and the small rest
__device__ __forceinline__ float residual(float a, float b, float c, float d, float rest) {
    float t, e1, e2, e3;
    two_sum32(a, -b, t, e1);
    two_sum32(t, -c, t, e2);
    two_sum32(t, -d, t, e3);
    return t + ((e1 + e2) + (e3 - rest));
}
// rest: what the pair leaves of the root
__device__ __forceinline__ dfl df_sqrt(dfl x, float& rest) {
    rest = 0.0f;
    if (!(x.hi > 0.0f)) return {0.0f, 0.0f};
    const float s = sqrtf(x.hi), g = 0.5f / s;
    const float c = (fmaf(-s, s, x.hi) + x.lo) * g, h = s + c, l = c - (h - s);
    const float p = h * h, d = 2.0f * h * l;
    const float r = residual(x.hi - p, fmaf(h, h, -p), -x.lo, d, fmaf(l, l, fmaf(2.0f * h, l, -d)));
    const float k = fmaf(r, g, l), y = h + k;
    rest = fmaf(r, g, l - k);
    return {y, k - (y - h)};
}
// 1 / (a + arest): of a root with its rest, so that 1/sqrt is rounded once
__device__ __forceinline__ dfl df_rcp_rounded(dfl a, float arest) {
    const float q = 1.0f / a.hi;
    const float c = q * fmaf(-a.lo, q, fmaf(-a.hi, q, 1.0f)), h = q + c, l = c - (h - q);
    const float p = a.hi * h, b = a.hi * l, d = a.lo * h;
    const float r = residual(1.0f - p, fmaf(a.hi, h, -p), b, d,
                             fmaf(arest, h, (fmaf(a.hi, l, -b) + fmaf(a.lo, h, -d)) + a.lo * l));
    const float k = fmaf(r, h, l), y = h + k;
    return {y, k - (y - h)};
}

// Lanczos on H = hopping + diag(d) from a fixed start vector, no
// re-orthogonalisation (the extreme Ritz values converge regardless), in
// double-float with the three Lanczos vectors in shared memory. The scalars of a
// step (alpha, beta, 1/beta) stay in double-float too, rounded as FP64 results would be
// (mean error of the bounds over 3096 chains of 43 lattices 2.2e-15, with FP64 scalars the same): as FP64
// numbers their square root, division and conversions, done by every warp, kept the
// narrow FP64 pipe busy for half of the kernel. Every 16
// steps each half of the CTA computes the smallest or largest eigenvalue of the
// Lanczos tridiagonal; the run stops when both moved less than 1e-13 of the
// spectral width in two consecutive checks, when the Krylov space is
// exhausted, or at kmax (then kStatusNoConverge). Writes (e_min, e_max, a, b)
// and the number of Lanczos steps.
// blockDim: 2 kRitzThreads .. kKpmThreads
__global__ void __launch_bounds__(kKpmThreads)
kpm_bounds_kernel(const KpmDesc* __restrict__ descs, const double* __restrict__ diag, int kmax,
                  KpmAB* __restrict__ ab, int* __restrict__ steps, float2* __restrict__ xdiag,
                  float2* __restrict__ xinv, int* __restrict__ status) {
    extern __shared__ __align__(16) double ksm[];
    const KpmDesc D = descs[blockIdx.x];
    const int n = D.n, tid = threadIdx.x;
    dfl* al = reinterpret_cast<dfl*>(ksm);
    dfl* b2 = al + kmax;
    dfl* V0 = b2 + kmax;  // three vectors and the diagonal, spacing ld
    dfl* V1 = V0 + D.ld;
    dfl* V2 = V1 + D.ld;
    dfl* dgd = V2 + D.ld;
    __shared__ float2 red[2][kKpmThreads / 32];
    int phase = 0;
    __shared__ float2 redd[kKpmThreads / 32];
    __shared__ double ext[2];
    __shared__ int slots[2][2][kRitzThreads / 32];
    const double* dg = diag + D.v_off;
    dfl s2 = {0.0f, 0.0f};
    for (int i = tid; i < n; i += blockDim.x) {
        const double x = (double)i * 0.6180339887498949;
        const dfl v = df_of(0.5 + (x - floor(x)));
        V1[i] = v;
        V0[i] = {0.0f, 0.0f};
        dgd[i] = df_of(dg[i]);
        s2 = df_add(s2, df_mul(v, v));
    }
    float rest;
    const dfl norm = df_sqrt(block_sum_df(s2, red, phase), rest), inv = df_rcp_rounded(norm, rest);
    for (int i = tid; i < n; i += blockDim.x) V1[i] = df_mul(V1[i], inv);
    __syncthreads();
    dfl bprev = {0.0f, 0.0f};
    float hnorm = 0.0f;
    double tmin = 0.0, tmax = 0.0, dmin = 0.0, dmax = 0.0;
    int stable = 0, kdim = 0;
    bool have_prev = false, done = false;
    for (int k = 0; k < kmax && !done; ++k) {
        const dfl nb = {-bprev.hi, -bprev.lo};
        dfl dot = {0.0f, 0.0f};
        for (int i = tid; i < n; i += blockDim.x) {
            dfl sacc = df_mul(dgd[i], V1[i]);
            for (int p = D.rowptr[i]; p < D.rowptr[i + 1]; ++p) {
                const float2 h = D.valf[p];
                sacc = df_add(sacc, df_mul({h.x, h.y}, V1[D.col[p]]));
            }
            const dfl w = df_add(sacc, df_mul(nb, V0[i]));
            V2[i] = w;
            dot = df_add(dot, df_mul(w, V1[i]));
        }
        const dfl alpha = block_sum_df(dot, red, phase);
        const dfl na = {-alpha.hi, -alpha.lo};
        dfl nn = {0.0f, 0.0f};
        for (int i = tid; i < n; i += blockDim.x) {
            const dfl w = df_add(V2[i], df_mul(na, V1[i]));
            V2[i] = w;
            nn = df_add(nn, df_mul(w, w));
        }
        const dfl beta2 = block_sum_df(nn, red, phase), beta = df_sqrt(beta2, rest);
        if (tid == 0) {
            al[k] = alpha;
            b2[k] = beta2;
        }
        hnorm = fmaxf(hnorm, fabsf(alpha.hi) + beta.hi + bprev.hi);
        kdim = k + 1;
        const bool exhausted = !(beta.hi > 1e-11f * hnorm);
        if (!exhausted) {
            const dfl ib = df_rcp_rounded(beta, rest);
            for (int i = tid; i < n; i += blockDim.x) V2[i] = df_mul(V2[i], ib);
        }
        __syncthreads();  // al/b2 and the new vector visible to all
        dfl* t = V0;
        V0 = V1;
        V1 = V2;
        V2 = t;
        bprev = beta;
        if (exhausted || (kdim >= 32 && kdim % 16 == 0) || kdim == kmax) {
            // Gershgorin bracket of the kdim x kdim tridiagonal (its last
            // off-diagonal b2[kdim-1] is the residual, not part of it)
            // in FP32 with a margin for its rounding
            float flo = 3e38f, fhi = -3e38f;
            for (int i = tid; i < kdim; i += blockDim.x) {
                const float r = (i > 0 ? sqrtf(b2[i - 1].hi) : 0.0f) + (i + 1 < kdim ? sqrtf(b2[i].hi) : 0.0f);
                flo = fminf(flo, al[i].hi - r);
                fhi = fmaxf(fhi, al[i].hi + r);
            }
            const float2 be = block_range(flo, fhi, redd);
            const double width = (double)be.y - (double)be.x, pad = 1e-6 * ((double)fabsf(be.x) + (double)fabsf(be.y)) + 1e-300;
            const double lo = (double)be.x - pad, hi = (double)be.y + pad;
            if (tid < 2 * kRitzThreads) {
                const int group = tid / kRitzThreads;
                const double span = fmax(4.0 * (group ? dmax : dmin), 1e-11 * width);
                const double e = ritz_extreme(al, b2, kdim, lo, hi, group ? tmax : tmin, span, have_prev, group,
                                              slots[group]);
                if ((tid & (kRitzThreads - 1)) == 0) ext[group] = e;
            }
            __syncthreads();
            const double nmin = ext[0], nmax = ext[1];
            __syncthreads();
            if (exhausted) {
                tmin = nmin;
                tmax = nmax;
                break;
            }
            const double tol = 1e-13 * fmax(nmax - nmin, fmax(fabs(nmin), fabs(nmax)));
            dmin = fabs(nmin - tmin);
            dmax = fabs(nmax - tmax);
            if (have_prev && dmin <= tol && dmax <= tol) {
                if (++stable >= 2) done = true;
            } else {
                stable = 0;
            }
            tmin = nmin;
            tmax = nmax;
            have_prev = true;
            if (!done && kdim == kmax && tid == 0) atomicOr(status, kStatusNoConverge);
        }
    }
    // x = (H - b) / a for the moments: its diagonal and 1/a, as FP32 pairs, once per chain
    const double a = (tmax - tmin) / 2., b = (tmax + tmin) / 2., inv_a = 1.0 / a;
    auto pair = [](double v) {
        const dfl d = df_of(v);
        return make_float2(d.hi, d.lo);
    };
    for (int i = tid; i < n; i += blockDim.x) xdiag[D.v_off + i] = pair(((D.hdiag[i] + dg[i]) + -b) * inv_a);
    if (tid == 0) {
        if (!(tmax - tmin == tmax - tmin)) atomicOr(status, kStatusNaN);
        xinv[blockIdx.x] = pair(inv_a);
        ab[blockIdx.x] = KpmAB{tmin, tmax, a, b};
        if (steps) steps[blockIdx.x] = kdim;
    }
}

// One warp per column j of T_m(x), m = 0..R, on the ball of radius R around
// j (local row 0 is j; rows in hop order, cnt[d] = rows within d hops).
// Writes, per column, tr[m] = (T_m(x))_jj, p1[m] = T_{m-1}(x)e_j . T_m(x)e_j and
// p2[m] = |T_m(x) e_j|^2 for m = 1..R at part[(v_off + j) * 3R + ...].
// What needs FP64 was made once per chain (xdiag, xinv), and the lanes share the
// conversions of the results: made row by row and result by result they took half
// of the kernel (256 x N = 576 1.05 -> 0.67 ms).
__global__ void kpm_moments_kernel(const KpmDesc* __restrict__ descs, const float2* __restrict__ xdiag,
                                   const float2* __restrict__ xinv, double* __restrict__ part, int wpc) {
    extern __shared__ __align__(16) double ksm[];
    const int c = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const KpmDesc D = descs[c];
    const int j = blockIdx.x * wpc + warp;
    if (j >= D.n) return;  // whole warps only; no block-wide barrier below
    const int R = D.R, nq = 3 * R;
    const int base = D.bptr[j], size = D.bptr[j + 1] - base;
    const int* cnt = D.bcnt + (size_t)j * (R + 1);
    // column vectors and the diagonal of x on the ball's rows, as FP32 pairs
    dfl* vp = reinterpret_cast<dfl*>(ksm) + (size_t)warp * 3 * D.bmax;
    dfl* vc = vp + D.bmax;
    dfl* xd = vc + D.bmax;
    const float2 iv = xinv[c];
    const dfl ia = {iv.x, iv.y};
    double* out = part + (size_t)(D.v_off + j) * nq;
    // result s = 3 (m - 1) + q is kept by lane s % 32 until 32 of them, or the last, are stored together
    dfl kept = {0.0f, 0.0f};
    int ns = 0;
    auto put = [&](dfl v) {
        if ((ns & 31) == lane) kept = v;
        if ((++ns & 31) == 0 || ns == nq) {
            const int s = ((ns - 1) & ~31) + lane;
            if (s < ns) out[(s % 3) * R + s / 3] = df_val(kept);
        }
    };
    for (int r = lane; r < size; r += 32) {
        const float2 x = xdiag[D.v_off + D.bsite[base + r]];
        xd[r] = {x.x, x.y};
        vp[r] = {r == 0 ? 1.0f : 0.0f, 0.0f};
        vc[r] = {0.0f, 0.0f};
    }
    __syncwarp();
    // x restricted to local row r: diagonal (H_ss - b)/a, off-diagonal H/a
    // (the off-diagonal sum is scaled by 1/a once), in double-float
    auto xrow = [&](int r, const dfl* v) {
        const int g = base + r;
        dfl off = {0.0f, 0.0f};
        for (int p = D.blrp[g]; p < D.blrp[g + 1]; ++p) {
            const float2 h = D.blv2[p];
            off = df_add(off, df_mul({h.x, h.y}, v[D.blcol[p]]));
        }
        return df_add(df_mul(off, ia), df_mul(xd[r], v[r]));
    };
    // T_1(x) e_j = x e_j on the rows within one hop
    dfl d2 = {0.0f, 0.0f};
    for (int r = lane; r < cnt[1]; r += 32) {
        const dfl v = xrow(r, vp);
        vc[r] = v;
        d2 = df_add(d2, df_mul(v, v));
    }
    __syncwarp();
    d2 = warp_sum_df(d2);
    put(vc[0]);  // tr[1]
    put(vc[0]);  // p1[1] = e_j . x e_j
    put(d2);     // p2[1]
    for (int m = 1; m < R; ++m) {
        // T_{m+1} e_j = 2 x T_m e_j - T_{m-1} e_j, written over T_{m-1} e_j
        const int rows = cnt[m + 1];
        for (int r = lane; r < rows; r += 32) {
            const dfl x = xrow(r, vc), o = vp[r];
            vp[r] = df_add({2.0f * x.hi, 2.0f * x.lo}, {-o.hi, -o.lo});
        }
        __syncwarp();
        dfl* t = vp;
        vp = vc;
        vc = t;
        dfl q1 = {0.0f, 0.0f}, q2 = {0.0f, 0.0f};
        for (int r = lane; r < rows; r += 32) {
            q1 = df_add(q1, df_mul(vp[r], vc[r]));
            q2 = df_add(q2, df_mul(vc[r], vc[r]));
        }
        q1 = warp_sum_df(q1);
        q2 = warp_sum_df(q2);
        put(vc[0]);
        put(q1);
        put(q2);
        __syncwarp();
    }
}

// Per chain: column sums, moments in the reference's order, coefficients,
// logZ. M moments (even), G grid points.
__global__ void __launch_bounds__(kKpmThreads)
kpm_final_kernel(const KpmDesc* __restrict__ descs, const double* __restrict__ part, const KpmAB* __restrict__ ab,
                 const double* __restrict__ beta_c, int M, int G, int mblk, double* __restrict__ mu_out,
                 double* __restrict__ logz, int* __restrict__ status) {
    extern __shared__ __align__(16) double ksm[];
    __shared__ double psum[kKpmThreads];
    const KpmDesc D = descs[blockIdx.x];
    const int R = D.R, nq = 3 * R, n = D.n, tid = threadIdx.x;
    double* sums = ksm;          // nq
    double* mu = sums + nq;      // M
    double* fg = mu + M;         // G: logz_f on the grid
    double* cm = fg + G;         // M: coefficients
    double* ac = cm + M;         // G: angles of the grid
    double* tab = ac + G;        // mblk x G: T_m on the grid
    // column sums: thread (g, q) adds every ng-th column (coalesced rows of nq), then
    // the ng partial sums in order
    const int ng = max(1, (int)blockDim.x / nq);
    for (int t = tid; t < nq * ng; t += blockDim.x) {
        const int q = t % nq;
        double s = 0.0;
        for (int j = t / nq; j < n; j += ng) s += part[(size_t)(D.v_off + j) * nq + q];
        if (ng == 1) sums[q] = s;
        else psum[t] = s;
    }
    if (ng > 1) {
        __syncthreads();
        if (tid < nq) {
            double s = psum[tid];
            for (int g = 1; g < ng; ++g) s += psum[g * nq + tid];
            sums[tid] = s;
        }
    }
    const KpmAB st = ab[blockIdx.x];
    const double a = st.a, b = st.b, beta = beta_c[blockIdx.x], N = (double)n;
    const double step = 1.0 / (double)(G - 1);
    for (int i = tid; i < G; i += blockDim.x) {
        const double x = -cos(M_PI * ((double)i * step));
        fg[i] = N * log(1. + exp(-beta * (a * x + b)));
    }
    __syncthreads();
    if (tid == 0) {
        // src/configuration.cpp:124-183: mu_1 from Tr x, mu_m (m <= M/2) from
        // the recursion unless set before, mu_{2m-1}, mu_{2m} from products
        // once 2m-1 >= M/2
        const double trx = sums[0];
        for (int m = 0; m < M; ++m) mu[m] = nan("");
        mu[0] = 1.0;
        if (M > 1) mu[1] = trx / N;
        for (int m = 2; m <= M / 2; ++m) {
            if (mu[m] != mu[m]) mu[m] = sums[m - 1] / N;
            int k = 2 * m - 1;
            if (k < M && k >= M / 2) {
                mu[k] = (sums[R + m - 1] * 2. - trx) / N;
                if (k != M - 1) {
                    ++k;
                    mu[k] = sums[2 * R + m - 1] / N * 2. - 1.0;
                }
            }
        }
    }
    // c_m = moment_f(logz_f, m): trapezoid in the angle (include/fk_mc/chebyshev.hpp:38-56).
    // T_m(x_i) = cos(m acos(x_i)) of the grid in parallel, then the sums (a thread
    // per moment evaluated six FP64 functions per grid interval before). acos(x_i)
    // once per point; the table goes in blocks of moments that fit its space.
    for (int i = tid; i < G; i += blockDim.x) ac[i] = acos(-cos(M_PI * ((double)i * step)));
    for (int m0 = 0; m0 < M; m0 += mblk) {
        const int mb = min(mblk, M - m0);
        __syncthreads();
        for (int q = tid; q < mb * G; q += blockDim.x) tab[q] = cos((double)(m0 + q / G) * ac[q % G]);
        __syncthreads();
        // a warp per moment on fine grids, whose blocks hold few moments: a thread each took 397 ms at M = 1024,
        // G = 4096
        const int per = G >= 64 ? 32 : 1, part = tid & (per - 1);
        for (int m = tid / per; m < mb; m += blockDim.x / per) {
            const double* t = tab + (size_t)m * G;
            double s = 0.0;
            for (int i = part; i + 1 < G; i += per)
                s += (fg[i + 1] * t[i + 1] + fg[i] * t[i]) * ((double)(i + 1) * step - (double)i * step);
            if (per > 1) s = warp_sum(s);
            if (part == 0) cm[m0 + m] = s * 0.5;
        }
    }
    __syncthreads();
    if (tid == 0) {
        double s = cm[0];
        for (int m = 1; m < M; ++m) s += 2. * cm[m] * mu[m];
        logz[blockIdx.x] = s;
        if (!(s - s == 0.0)) atomicOr(status, kStatusNaN);
        if (mu_out)
            for (int m = 0; m < M; ++m) mu_out[(size_t)blockIdx.x * M + m] = mu[m];
    }
}

}  // namespace

size_t kpm_moment_smem_bytes(int bmax, int wpc) { return sizeof(double) * 3 * (size_t)bmax * wpc; }

int kpm_warps_per_cta(int bmax) {
    const size_t per = sizeof(double) * 3 * (size_t)bmax;
    int w = (int)((96 * 1024) / per);
    return w < 1 ? 1 : (w > 8 ? 8 : w);
}

cudaError_t launch_kpm(const KpmDesc* d_kdesc, int batch, int max_n, int max_ld, int max_bmax, int R, int M, int G,
                       int kmax, const double* d_diag, const double* d_beta, KpmAB* d_ab, int* d_steps,
                       double* d_part, float2* d_xdiag, float2* d_xinv, double* d_mu, double* d_logz, int* d_status,
                       cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    if (batch > 65535) return cudaErrorInvalidValue;  // grid y limit of the moment kernel
    cudaError_t err;
    const size_t sm_b = sizeof(dfl) * (2 * (size_t)kmax + 4 * (size_t)max_ld);
    if ((err = allow_smem<kpm_bounds_kernel>())) return err;
    // the threads that share the rows evenly: 256 for N = 576 left a third of them idle in the last pass, and for
    // N = 144 barriers for warps without rows (512 chains of N = 144 2.61 -> 2.47 ms for three steps)
    const int passes = (max_n + kKpmThreads - 1) / kKpmThreads;
    const int bt = max(2 * kRitzThreads, ((max_n + passes - 1) / passes + 31) / 32 * 32);
    kpm_bounds_kernel<<<batch, bt, sm_b, st>>>(d_kdesc, d_diag, kmax, d_ab, d_steps, d_xdiag, d_xinv, d_status);
    if ((err = cudaGetLastError())) return err;
    const int wpc = kpm_warps_per_cta(max_bmax);
    const size_t sm_m = kpm_moment_smem_bytes(max_bmax, wpc);
    if ((err = allow_smem<kpm_moments_kernel>())) return err;
    kpm_moments_kernel<<<dim3((max_n + wpc - 1) / wpc, batch), 32 * wpc, sm_m, st>>>(d_kdesc, d_xdiag, d_xinv, d_part,
                                                                                      wpc);
    if ((err = cudaGetLastError())) return err;
    // moments per block of the T_m table: as many as fit in 64 KB
    const int mblk = max(1, min(M, (int)(8192 / G)));
    const size_t sm_f = sizeof(double) * (3 * (size_t)R + 2 * (size_t)M + (2 + (size_t)mblk) * (size_t)G);
    if ((err = allow_smem<kpm_final_kernel>())) return err;
    kpm_final_kernel<<<batch, kKpmThreads, sm_f, st>>>(d_kdesc, d_part, d_ab, d_beta, M, G, mblk, d_mu, d_logz,
                                                     d_status);
    return cudaGetLastError();
}

}  // namespace fkg
