// trieig.cu — eigenvalues (and, for the mixed path and calc_ed(true),
// eigenvectors) of the symmetric tridiagonal T = tridiag(e, d, e).
//
// Replaces the tridiagonal QR half of Eigen::SelfAdjointEigenSolver used at
// src/configuration.cpp:213. The eigenvalues are computed in FP64 and come
// out ascending (src/measures/spectrum.cpp:13-21 relies on the order).
//
// GB300's FP64 pipe runs at about 1/58 of its FP32 pipe, so the eigenvalue
// search spends as little FP64 work as possible while staying FP64-accurate:
//   1. FP32 bisection on Sturm counts of the FP32-rounded T isolates each
//      eigenvalue to an interval of width ~ 4 eps32 ||T||.  Kahan's analysis
//      of the Sturm recurrence makes each FP32 count exact for a matrix
//      within a few eps32 ||T|| of T, so widening by 16 eps32 ||T|| gives a
//      bracket of the FP64 eigenvalue;
//   2. where the widened brackets of the neighbouring indices j-1 and j+1
//      stay clear of it, or FP32 counts further out say so (block edges), that
//      bracket holds exactly lambda_j;
//   3. if the bracket holds exactly one eigenvalue, Newton on the characteristic
//      polynomial p_n(x) = det(T - x I) (three-term recurrence, rescaled by
//      powers of two, no divisions) in double-float and one last step with
//      p_n in FP64, two where a neighbour is so close that the pairs'
//      derivative is not good enough;
//   4. otherwise (eigenvalues closer than the FP32 resolution) FP64 Sturm counts
//      at the ends, then safeguarded Newton in FP64, or bisection (multisection
//      where a warp has lanes to spare).
// One thread per eigenvalue index; d and e of the chain sit in shared memory.
#include <cfloat>

#include "fkg_common.cuh"

namespace fkg {
namespace {

constexpr int kEigThreads = 128;

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// FP32 Sturm count: eigenvalues of T below x, from q_0 = d_0 - x,
// q_k = (d_k - x) - e_{k-1}^2 / q_{k-1}, counting the q_k with the sign bit
// set. de[k] = (d_k, e_{k-1}^2). The approximate reciprocal perturbs each
// e^2 by a relative 2^-22 at most. A zero q_k makes q_{k+1} an infinity of
// the opposite sign and q_{k+2} = d_{k+2} - x again (IEEE arithmetic; e^2 is
// floored at FLT_MIN so that 0 x inf cannot occur), which counts exactly one
// negative between them for either sign of the zero.
__device__ __forceinline__ int count32(const float2* __restrict__ de, int n, float x) {
    float q = de[0].x - x;
    int c = __float_as_uint(q) >> 31;
    for (int i = 1; i < n; ++i) {
        const float2 v = de[i];
        q = fmaf(-v.y, rcp_approx(q), v.x - x);
        c += __float_as_uint(q) >> 31;
    }
    return c;
}

// Number of eigenvalues below x: sign changes of the Sturm sequence
// p_0 = 1, p_k = (d_k - x) p_{k-1} - e_{k-1}^2 p_{k-2} (division-free
// projective form of q_k = p_k / p_{k-1}; rescaled by powers of two, which
// keeps every sign). A zero p_k is replaced by -pivmin p_{k-1}, i.e.
// q_k = -pivmin, the usual pivot floor of Sturm counting.
__device__ __forceinline__ int count64(const double* __restrict__ d, const double* __restrict__ e2, int n, double x,
                                       double pivmin) {
    double p0 = 1.0;
    double p1 = d[0] - x;
    if (p1 == 0.0) p1 = -pivmin;
    int c = p1 < 0.0;
    for (int i = 1; i < n; ++i) {
        double p2 = fma(d[i] - x, p1, -e2[i - 1] * p0);
        if (p2 == 0.0) p2 = -pivmin * p1;
        c += (__double2hiint(p2) ^ __double2hiint(p1)) < 0;
        p0 = p1;
        p1 = p2;
        if ((i & 7) == 0) {
            const double m = fmax(fabs(p0), fabs(p1));
            if (m > 0x1p400) { p0 *= 0x1p-400; p1 *= 0x1p-400; }
            else if (m < 0x1p-400) { p0 *= 0x1p400; p1 *= 0x1p400; }
        }
    }
    return c;
}

// p_n(x) and p_n'(x) up to a common positive power-of-two scale.
__device__ __forceinline__ void charpoly(const double* __restrict__ d, const double* __restrict__ e2, int n,
                                         double x, double& p, double& dp) {
    double p0 = 1.0, dp0 = 0.0;          // p_{k-1}, p'_{k-1}
    double p1 = d[0] - x, dp1 = -1.0;    // p_k, p'_k
    for (int i = 1; i < n; ++i) {
        const double t = d[i] - x, b = e2[i - 1];
        const double p2 = fma(t, p1, -b * p0);
        const double dp2 = fma(t, dp1, fma(-b, dp0, -p1));
        p0 = p1; dp0 = dp1; p1 = p2; dp1 = dp2;
        if ((i & 7) == 0) {
            const double m = fmax(fabs(p1), fabs(dp1));
            if (m > 0x1p400) { p0 *= 0x1p-400; dp0 *= 0x1p-400; p1 *= 0x1p-400; dp1 *= 0x1p-400; }
            else if (m < 0x1p-400 && m > 0.0) { p0 *= 0x1p400; dp0 *= 0x1p400; p1 *= 0x1p400; dp1 *= 0x1p400; }
        }
    }
    p = p1;
    dp = dp1;
}

// 2^k, -1022 <= k <= 1023
__device__ __forceinline__ double pow2(int k) { return __hiloint2double((1023 + k) << 20, 0); }

struct TriShared {
    double* d;
    double* e2;
    float* d32;
    float* e232;  // e_i^2 in FP32, floored at FLT_MIN (i < n - 1)
    float2* de;   // (d_i, e_{i-1}^2) for the FP32 counts
    float* e2l;   // e_i^2 - e232[i]
    float* dl;    // d_i - d32[i] (null: T is FP32-exact)
    int k;        // d32, dl and e232, e2l hold 2^-k T (0 unless with dl and ||T|| is far from 1)
};

// shared-memory layout of one chain's tridiagonal (pairs: d as FP32 pairs too)
__device__ __forceinline__ TriShared tri_shared(double* sm, int ld, bool pairs) {
    float* f = (float*)(sm + 2 * ld);
    return TriShared{sm, sm + ld, f, f + ld, (float2*)(f + 2 * ld), f + 4 * ld, pairs ? f + 5 * ld : nullptr, 0};
}

// Loads d, e^2 (FP64 and FP32 copies) of chain D into shared memory and
// returns the Gershgorin interval, max e^2 and the norm estimate.
__device__ void load_tridiag(const ChainDesc& D, const double* __restrict__ dd, const double* __restrict__ ee,
                             TriShared& S, double& gl, double& gu, double& emax2) {
    const int n = D.n;
    __shared__ double red[3][kEigThreads / 32];
    gl = DBL_MAX; gu = -DBL_MAX; emax2 = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double di = dd[D.v_off + i];
        const double el = i > 0 ? fabs(ee[D.v_off + i - 1]) : 0.0;
        const double er = i + 1 < n ? fabs(ee[D.v_off + i]) : 0.0;
        S.d[i] = di;
        S.e2[i] = er * er;
        S.d32[i] = (float)di;
        S.e232[i] = i + 1 < n ? fmaxf((float)(er * er), FLT_MIN) : 0.f;
        S.e2l[i] = (float)(er * er - (double)S.e232[i]);
        if (S.dl) S.dl[i] = (float)(di - (double)S.d32[i]);
        S.de[i] = make_float2((float)di, i > 0 ? fmaxf((float)(el * el), FLT_MIN) : 0.f);
        gl = fmin(gl, di - el - er);
        gu = fmax(gu, di + el + er);
        emax2 = fmax(emax2, er * er);
    }
    gl = warp_min(gl);
    gu = warp_max(gu);
    emax2 = warp_max(emax2);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) { red[0][wid] = gl; red[1][wid] = gu; red[2][wid] = emax2; }
    __syncthreads();
    gl = red[0][0]; gu = red[1][0]; emax2 = red[2][0];
    for (int q = 1; q < (int)(blockDim.x / 32); ++q) {
        gl = fmin(gl, red[0][q]); gu = fmax(gu, red[1][q]); emax2 = fmax(emax2, red[2][q]);
    }
    if (!S.dl) return;
    // The pairs' recurrence is rescaled every four rows, by at most 2^50: away from norms around 1 it would leave
    // FP32's range in between, and every eigenvalue go to the FP64 list.
    const double tnorm = fmax(fabs(gl), fabs(gu));
    if ((tnorm >= 0.25 && tnorm < 32.0) || !(tnorm >= 0x1p-480 && tnorm <= 0x1p480)) return;
    S.k = ilogb(tnorm);
    const double sc = pow2(-S.k), sc2 = pow2(-2 * S.k);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double di = S.d[i] * sc, e2 = S.e2[i] * sc2;
        S.d32[i] = (float)di;
        S.dl[i] = (float)(di - (double)S.d32[i]);
        S.e232[i] = i + 1 < n ? fmaxf((float)e2, FLT_MIN) : 0.f;
        S.e2l[i] = (float)(e2 - (double)S.e232[i]);
    }
}

// Derived bounds of one chain's tridiagonal: the norm estimate, the pivot
// floor and the Gershgorin interval widened by the rounding of the counts.
struct TriBounds {
    double gl, gu, tnorm, pivmin;
};

__device__ __forceinline__ TriBounds tri_bounds(int n, double gl, double gu, double emax2) {
    TriBounds B;
    B.tnorm = fmax(fabs(gl), fabs(gu));
    B.pivmin = DBL_MIN * fmax(1.0, emax2);
    B.gl = gl - (2.0 * DBL_EPSILON * B.tnorm * n + 4.0 * B.pivmin);
    B.gu = gu + (2.0 * DBL_EPSILON * B.tnorm * n + 4.0 * B.pivmin);
    return B;
}

// Step 1: FP32 brackets [lo, hi] of the block's eigenvalues j (all threads
// of the block call this). Two rounds of multisection narrow the start: the
// block's threads count at 128 evenly spaced points, first over the
// Gershgorin interval, then over the span of the block's own eigenvalues,
// and each thread takes the pair of neighbouring points whose counts enclose
// its index (a binary search for the first count above j, which keeps
// count(lo) <= j < count(hi) whether or not the FP32 counts are monotone);
// bisection finishes.
__device__ void block_brackets(const TriShared& S, int n, int j, bool active, const TriBounds& B, float& lo,
                               float& hi) {
    __shared__ int cs[kEigThreads];
    __shared__ float span[2];
    const int t = threadIdx.x, T = blockDim.x;
    const float t32 = (float)B.tnorm;
    const float L0 = fminf((float)B.gl, (float)B.gl - 4.f * FLT_EPSILON * t32);
    const float R0 = fmaxf((float)B.gu, (float)B.gu + 4.f * FLT_EPSILON * t32);
    float L = L0, R = R0;
    lo = L0;
    hi = R0;
    const int jfirst = blockIdx.y * T, jlast = min(n - 1, jfirst + T - 1);
    for (int round = 0; round < 2; ++round) {
        const float h = (R - L) / (float)T;
        cs[t] = count32(S.de, n, t + 1 < T ? L + (float)(t + 1) * h : R);
        __syncthreads();
        if (active) {
            int a = 0, b = T;  // first index with cs > j
            while (a < b) {
                const int m = (a + b) >> 1;
                if (cs[m] > j) b = m; else a = m + 1;
            }
            if (a < T) {
                const float nlo = a == 0 ? L : L + (float)a * h;
                const float nhi = a + 1 < T ? L + (float)(a + 1) * h : R;
                if (nlo < nhi) { lo = nlo; hi = nhi; }
            }
            if (j == jfirst) span[0] = lo;
            if (j == jlast) span[1] = hi;
        }
        __syncthreads();
        L = span[0];
        R = span[1];
        if (!(L < R)) break;  // uniform: every thread read the same span
    }
    if (!active) return;
    for (int it = 0; it < 64; ++it) {
        const float mid = 0.5f * (lo + hi);
        if (hi - lo <= 4.f * FLT_EPSILON * fmaxf(fabsf(lo), fabsf(hi)) + FLT_EPSILON * t32 || mid <= lo || mid >= hi) break;
        if (count32(S.de, n, mid) > j) hi = mid;
        else lo = mid;
    }
}

// Half-width of the band around an FP32 bracket that is sure to hold the
// eigenvalue: Kahan's analysis makes each FP32 count exact for a matrix
// within a few eps32 ||T|| of T.
__device__ __forceinline__ double bracket_slack(const TriBounds& B) { return 16.0 * FLT_EPSILON * B.tnorm; }

// Safeguarded Newton on p_n in FP64 inside [a, b], which holds exactly one
// eigenvalue, number ca; sign(p_n(x)) = (-1)^count(x). Converged when the step
// falls below 4 eps max(|x|, ||T||), i.e. at the accuracy of the Sturm
// recurrence itself; from the FP32 bracket that takes 3-5 evaluations, the cap
// of 12 only stops rounding-level oscillation.
// A Newton step s_k after s_{k-1} leaves an error of about |s_k|^2 |p''/2p'| ~
// |s_k|^3 / s_{k-1}^2 (quadratic convergence); when that is 4x below the
// tolerance the step is the last one, which from an FP32 bracket usually saves
// the third evaluation.
__device__ double newton64(const TriShared& S, int n, int ca, double tnorm, double a, double b) {
    const double eps = DBL_EPSILON;
    const double sa = (ca & 1) ? -1.0 : 1.0;  // sign of p_n at a
    double x = 0.5 * (a + b), dxold = b - a, dx = dxold, prev = 0.0;
    for (int it = 0; it < 12; ++it) {
        double p, dp;
        charpoly(S.d, S.e2, n, x, p, dp);
        if (p == 0.0) { a = b = x; break; }
        if ((p > 0.0) == (sa > 0.0)) a = x; else b = x;
        const double step = p / dp;
        const double tol = 4.0 * eps * fmax(fabs(x), tnorm);
        // converged: the Newton correction is at the rounding level of p_n,
        // or the one after it would be
        if (dp != 0.0 && (fabs(step) <= tol || (prev > 0.0 && fabs(step) * step * step <= 0.25 * tol * prev * prev)) &&
            x - step >= a && x - step <= b) {
            x -= step;
            break;
        }
        double xn = x - step;
        if (!(dp != 0.0) || !(xn > a && xn < b) || fabs(2.0 * (xn - x)) > fabs(dxold)) {
            dxold = dx;
            xn = 0.5 * (a + b);
            dx = xn - x;
            prev = 0.0;
        } else {
            dxold = dx;
            dx = xn - x;
            prev = fabs(step);
        }
        x = xn;
        if (fabs(dx) <= 4.0 * eps * fmax(fabs(x), tnorm) || b - a <= 4.0 * eps * fmax(fabs(x), tnorm)) break;
    }
    return fmin(fmax(x, a), b);
}

// FP64 eigenvalue j of a bracket that nothing confirms yet, by a group of p
// lanes (p a power of two, the group's lanes adjacent; `active`: the group has
// an eigenvalue; a whole warp calls): Sturm counts at both ends; if it holds
// exactly lambda_j Newton, else multisection with p points a round (p = 1:
// bisection).
__device__ double refine64_group(const TriShared& S, int n, int j, const TriBounds& B, float lo, float hi, int p,
                                 bool active, int* status) {
    const double eps = DBL_EPSILON;
    const int lane = threadIdx.x & 31, k = lane & (p - 1), base = lane - k;
    const unsigned group = p == 32 ? 0xffffffffu : (1u << p) - 1;
    const double delta = bracket_slack(B);
    double a = fmax((double)lo - delta, B.gl), b = fmin((double)hi + delta, B.gu);
    int ca = active ? count64(S.d, S.e2, n, k == 0 ? a : b, B.pivmin) : 0, cb;
    if (p == 1) {
        cb = active ? count64(S.d, S.e2, n, b, B.pivmin) : 0;
    } else {
        cb = __shfl_sync(0xffffffffu, ca, base + 1);
        ca = __shfl_sync(0xffffffffu, ca, base);
    }
    if (!(ca <= j && j < cb)) {
        a = B.gl; b = B.gu; ca = 0; cb = n;
    }
    const bool newton = active && ca == j && cb == j + 1;
    bool run = active && !newton;
    for (int it = 0; it < 128; ++it) {
        const double w = b - a, mid = 0.5 * (a + b);
        if (w <= 2.0 * eps * fmax(fabs(a), fabs(b)) + 0.5 * eps * B.tnorm || mid <= a || mid >= b) run = false;
        if (!__any_sync(0xffffffffu, run)) break;
        const double x = p == 1 ? mid : fmin(fmax(a + w * ((double)(k + 1) / (p + 1)), a), b);
        const bool above = run && count64(S.d, S.e2, n, x, B.pivmin) > j;
        const unsigned up = __ballot_sync(0xffffffffu, above) >> base & group;
        const int f = up ? __ffs(up) - 1 : p;  // first point above lambda_j
        const double nb = __shfl_sync(0xffffffffu, x, base + min(f, p - 1));
        const double na = __shfl_sync(0xffffffffu, x, base + max(f - 1, 0));
        if (run && f < p) b = nb;
        if (run && f > 0) a = na;
        if (it == 127 && run) atomicOr(status, kStatusNoConverge);
    }
    return newton ? newton64(S, n, ca, B.tnorm, a, b) : 0.5 * (a + b);
}

// Gaps between the widened FP32 bracket of this thread's eigenvalue and its
// neighbours' (same block; +inf at the ends of the spectrum, -1 where the
// neighbour belongs to another block). br: 2 floats per thread, shared.
__device__ __forceinline__ void neighbour_gaps(float* br, int n, int j, bool active, float lo, float hi,
                                               double delta, double& gl_gap, double& gr_gap) {
    const int t = threadIdx.x;
    br[2 * t] = lo;
    br[2 * t + 1] = hi;
    __syncthreads();
    gl_gap = -1.0;
    gr_gap = -1.0;
    if (!active) return;
    if (j == 0) gl_gap = DBL_MAX;
    else if (t > 0) gl_gap = ((double)lo - delta) - ((double)br[2 * (t - 1) + 1] + delta);
    if (j == n - 1) gr_gap = DBL_MAX;
    else if (t + 1 < (int)blockDim.x) gr_gap = ((double)br[2 * (t + 1)] - delta) - ((double)hi + delta);
}

// ---- mixed path: the eigenvalues of T only serve as shifts of the FP32
// twisted factorisation (the final eigenvalues are FP64 Rayleigh quotients
// with H). T comes from the FP32 reduction, so d_i and e_i are FP32 numbers
// and e_i^2 is exactly the FP32 pair e2h + e2l. The shifts are refined in
// double-float arithmetic (an unevaluated FP32 pair, ~48 significant bits),
// which GB300 runs about ten times faster than FP64: the FP32 bracket, then
// safeguarded Newton on p_n in double-float (p_n'(x) in FP32 is accurate
// enough for the step); converged at 1e-13 ||T||, far below what the FP32
// twisted factorisation can resolve. FP64 (list64) remains for the brackets
// that the double-float Sturm counts cannot confirm: none for random
// configurations, all of them where every eigenvalue belongs to a multiplet.

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float v = s - a;
    e = (a - (s - v)) + (b - v);
}
__device__ __forceinline__ void fast_two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    e = b - (s - a);
}

// One step of p_k = (d_k - x) p_{k-1} - e_{k-1}^2 p_{k-2} in double-float.
struct DfRow {
    float th, tl;  // d_k - x as a pair
};
__device__ __forceinline__ DfRow df_shift(float dk, float xh, float xl) {
    DfRow r;
    float e;
    two_sum(dk, -xh, r.th, e);
    r.tl = e - xl;
    return r;
}
__device__ __forceinline__ void df_step(const DfRow& t, float bh, float bl, float p1h, float p1l, float p0h,
                                        float p0l, float& p2h, float& p2l) {
    const float ah = t.th * p1h;
    const float al = fmaf(t.th, p1l, fmaf(t.tl, p1h, fmaf(t.th, p1h, -ah)));
    const float ch = bh * p0h;
    const float cl = fmaf(bh, p0l, fmaf(bl, p0h, fmaf(bh, p0h, -ch)));
    float sh, se;
    two_sum(ah, -ch, sh, se);
    fast_two_sum(sh, se + (al - cl), p2h, p2l);
}
// power-of-two rescaling of the recurrence state (keeps every sign and ratio)
__device__ __forceinline__ float df_scale(float m) {
    return m > 0x1p50f ? 0x1p-50f : (m < 0x1p-50f && m > 0.f ? 0x1p50f : 1.f);
}

// p_n(x) (pair, up to a positive power-of-two scale) and p_n'(x) (FP32, same scale)
__device__ void charpoly_df(const float* __restrict__ d, const float* __restrict__ e2h,
                            const float* __restrict__ e2l, int n, float xh, float xl, float& ph, float& pl,
                            float& dp) {
    float p0h = 1.f, p0l = 0.f, dp0 = 0.f;
    DfRow t = df_shift(d[0], xh, xl);
    float p1h, p1l;
    fast_two_sum(t.th, t.tl, p1h, p1l);
    float dp1 = -1.f;
    for (int i = 1; i < n; ++i) {
        t = df_shift(d[i], xh, xl);
        float p2h, p2l;
        df_step(t, e2h[i - 1], e2l[i - 1], p1h, p1l, p0h, p0l, p2h, p2l);
        const float dp2 = fmaf(t.th, dp1, -fmaf(e2h[i - 1], dp0, p1h));
        p0h = p1h; p0l = p1l; dp0 = dp1;
        p1h = p2h; p1l = p2l; dp1 = dp2;
        if ((i & 3) == 0) {
            const float sc = df_scale(fmaxf(fabsf(p1h), fabsf(dp1)));
            p0h *= sc; p0l *= sc; dp0 *= sc; p1h *= sc; p1l *= sc; dp1 *= sc;
        }
    }
    ph = p1h;
    pl = p1l;
    dp = dp1;
}

// Sturm count at x in double-float: sign changes of p_0 = 1, p_1, ..., p_n (a
// zero p_k counts as the sign opposite to p_{k-1}, i.e. as negative for q_k).
__device__ int count_df(const float* __restrict__ d, const float* __restrict__ e2h, const float* __restrict__ e2l,
                        int n, float xh, float xl) {
    float p0h = 1.f, p0l = 0.f;
    DfRow t = df_shift(d[0], xh, xl);
    float p1h, p1l;
    fast_two_sum(t.th, t.tl, p1h, p1l);
    int c = !(p1h > 0.f);
    for (int i = 1; i < n; ++i) {
        t = df_shift(d[i], xh, xl);
        float p2h, p2l;
        df_step(t, e2h[i - 1], e2l[i - 1], p1h, p1l, p0h, p0l, p2h, p2l);
        const bool neg = p2h == 0.f ? (p1h > 0.f) : ((p2h > 0.f) != (p1h > 0.f));
        c += neg;
        if (p2h == 0.f) p2h = p1h > 0.f ? -0x1p-100f : 0x1p-100f;  // sign opposite to p_{k-1}
        p0h = p1h; p0l = p1l;
        p1h = p2h; p1l = p2l;
        if ((i & 3) == 0) {
            const float sc = df_scale(fabsf(p1h) + fabsf(p0h));
            p0h *= sc; p0l *= sc; p1h *= sc; p1l *= sc;
        }
    }
    return c;
}

constexpr int kDfIters = 6;

// Shift j from its FP32 bracket in double-float; false when the bracket or the
// iteration cannot be trusted (then FP64 decides).
__device__ bool shift_df(const float* d, const float* e2h, const float* e2l, int n, int j, const TriBounds& B,
                         float lo, float hi, bool isolated, double& out) {
    const double delta = bracket_slack(B);
    const double a0 = fmax((double)lo - delta, B.gl), b0 = fmin((double)hi + delta, B.gu);
    double a = a0, b = b0;
    int ca = j;
    if (!isolated) {
        const float ah = (float)a, al = (float)(a - (double)ah), bh = (float)b, bl = (float)(b - (double)bh);
        ca = count_df(d, e2h, e2l, n, ah, al);
        const int cb = count_df(d, e2h, e2l, n, bh, bl);
        if (!(ca == j && cb == j + 1)) return false;
    }
    const bool neg_at_a = ca & 1;  // sign of p_n at a is (-1)^count
    const double tol = 1e-13 * B.tnorm;
    float xh = 0.5f * (lo + hi), xl = 0.5f * (lo + hi) - xh;
    xl = (float)(0.5 * ((double)lo + (double)hi) - (double)xh);
    float prev = 0.f;
    for (int it = 0; it < kDfIters; ++it) {
        float ph, pl, dp;
        charpoly_df(d, e2h, e2l, n, xh, xl, ph, pl, dp);
        const double x = (double)xh + (double)xl;
        const float p = ph + pl;
        if (p == 0.f) { out = x; return true; }
        if ((p < 0.f) == neg_at_a) a = x; else b = x;
        if (!(dp != 0.f) || !isfinite(p / dp)) return false;
        const float step = p / dp;
        float sh, se;
        two_sum(xh, -step, sh, se);
        float nh, nl;
        fast_two_sum(sh, se + xl, nh, nl);
        const double xn = (double)nh + (double)nl;
        if (!(xn >= a0 && xn <= b0)) return false;
        const float as = fabsf(step);
        if ((double)as <= tol || (prev > 0.f && (double)as * as * as <= 0.25 * tol * (double)prev * prev)) {
            out = xn;
            return true;
        }
        prev = as;
        xh = nh;
        xl = nl;
    }
    return false;
}

// The listed eigenvalues in FP64. A warp's FP64 instruction costs the narrow pipe
// the same for one lane as for 32, so eigenvalues share a warp: in ordered
// configurations all of them belong to multiplets and are listed, and a warp for
// each took 243 ms for 256 checkerboards of N = 576 (37 now). A short list gets
// more lanes an eigenvalue, whose rounds are fewer (32 lanes 7, 4 lanes 15, one 35), as
// far as two warps reach (128 chains of cubic3d L = 8 with 5 % defects 8.9 ms with one
// warp, 9.3 with two, 9.9 with four; 64 of cubic1d L = 343 1.28, 1.10, 0.98). The number of
// lanes changes an eigenvalue's last bits, so it depends on nothing but the list.
// A function of its own, as last_step, with its arguments by value: inlined, they
// cost the kernels' FP32 recurrences 5 % (16 chains of N = 576 0.505 -> 0.480 ms mixed).
__device__ __noinline__ void list64(const ChainDesc D, const TriShared S, int n, const TriBounds B, int count, const int* list,
                       const float* lbr, double* __restrict__ ww, int* __restrict__ status) {
    if (count == 0) return;
    int p = 1;
    while (p < 32 && 2 * p * count <= 64) p *= 2;
    if ((int)(threadIdx.x & ~31u) / p >= count) return;  // nothing for this warp
    const int q = threadIdx.x / p, i = min(q, count - 1);
    const double lam = refine64_group(S, n, list[i], B, lbr[2 * i], lbr[2 * i + 1], p, q < count, status);
    if (q < count && (threadIdx.x & (p - 1)) == 0) {
        ww[D.v_off + list[i]] = lam;
        if (!isfinite(lam)) atomicOr(status, kStatusNaN);
    }
}

// p_n and p_n' as charpoly_df with d and e^2 as pairs; `e`: the common scale is 2^e.
__device__ void charpoly_df2(const TriShared& S, int n, float xh, float xl, float& p, float& dp, int& e) {
    float p0h = 1.f, p0l = 0.f, dp0 = 0.f;
    DfRow t = df_shift(S.d32[0], xh, xl - S.dl[0]);
    float p1h, p1l;
    fast_two_sum(t.th, t.tl, p1h, p1l);
    float dp1 = -1.f;
    e = 0;
    for (int i = 1; i < n; ++i) {
        t = df_shift(S.d32[i], xh, xl - S.dl[i]);
        const float bh = S.e232[i - 1];
        float p2h, p2l;
        df_step(t, bh, S.e2l[i - 1], p1h, p1l, p0h, p0l, p2h, p2l);
        const float dp2 = fmaf(t.th, dp1, -fmaf(bh, dp0, p1h));
        p0h = p1h; p0l = p1l; dp0 = dp1;
        p1h = p2h; p1l = p2l; dp1 = dp2;
        if ((i & 3) == 0) {
            const float m = fmaxf(fabsf(p1h), fabsf(dp1));
            const float sc = df_scale(m);
            e += m > 0x1p50f ? 50 : (m < 0x1p-50f && m > 0.f ? -50 : 0);
            p0h *= sc; p0l *= sc; dp0 *= sc; p1h *= sc; p1l *= sc; dp1 *= sc;
        }
    }
    p = p1h + p1l;
    dp = dp1;
}

// Newton in double-float from the middle of an isolated FP32 bracket, until the
// next step would be below 1e-13 ||T||; returns the point, and the derivative of
// 2^-k T's polynomial there (to FP32 accuracy, up to 2^edp). False when the
// iteration cannot be trusted.
__device__ bool newton_df(const TriShared& S, int n, const TriBounds& B, float lo, float hi, double& x, double& dpx,
                          int& edp) {
    const double delta = bracket_slack(B), sc = pow2(-S.k), tol = 1e-13 * B.tnorm * sc;
    const double a = ((double)lo - delta) * sc, b = ((double)hi + delta) * sc, x0 = 0.5 * ((double)lo + (double)hi) * sc;
    float xh = (float)x0, xl = (float)(x0 - (double)xh), prev = 0.f;
    for (int it = 0; it < kDfIters; ++it) {
        float p, dp;
        charpoly_df2(S, n, xh, xl, p, dp, edp);
        const float step = p / dp;
        if (!(dp != 0.f) || !isfinite(dp) || !isfinite(step)) return false;
        float sh, se, nh, nl;
        two_sum(xh, -step, sh, se);
        fast_two_sum(sh, se + xl, nh, nl);
        x = (double)nh + (double)nl;
        if (!(x >= a && x <= b)) return false;
        const float as = fabsf(step);
        if ((double)as <= tol || (prev > 0.f && (double)as * as * as <= 0.25 * tol * (double)prev * prev)) {
            dpx = (double)dp;
            x *= pow2(S.k);
            return true;
        }
        prev = as;
        xh = nh;
        xl = nl;
    }
    return false;
}

// Does the widened bracket [lo - delta, hi + delta] hold exactly lambda_j, with no
// other eigenvalue within (m - 2) delta of it? Decided with FP32 counts m delta out:
// an FP32 count at y is the exact count at a point within delta of y, so count32(lo
// - m delta) >= j puts lambda_{j-1} below lo - (m - 1) delta, and likewise above.
__device__ __forceinline__ bool isolated32(const TriShared& S, int n, int j, const TriBounds& B, float lo, float hi,
                                           double m) {
    const float out = (float)(m * bracket_slack(B));
    return (j == 0 || count32(S.de, n, lo - out) >= j) && (j == n - 1 || count32(S.de, n, hi + out) <= j + 1);
}

// p_n(x) in FP64 up to 2^e (no derivative: three FP64 operations a row).
__device__ __forceinline__ double charpoly_value(const double* __restrict__ d, const double* __restrict__ e2, int n,
                                                 double x, int& e) {
    double p0 = 1.0, p1 = d[0] - x;
    e = 0;
    for (int i = 1; i < n; ++i) {
        const double p2 = fma(d[i] - x, p1, -e2[i - 1] * p0);
        p0 = p1;
        p1 = p2;
        if ((i & 7) == 0) {
            // magnitude from the exponent fields: the FP64 pipe is the bound here
            const int m = max(__double2hiint(p0) & 0x7ff00000, __double2hiint(p1) & 0x7ff00000);
            if (m > (1023 + 400) << 20) { p0 *= 0x1p-400; p1 *= 0x1p-400; e += 400; }
            else if (m < (1023 - 400) << 20 && m > 0) { p0 *= 0x1p400; p1 *= 0x1p400; e -= 400; }
        }
    }
    return p1;
}

// The last step: from x (an FP32-pair Newton point of the eigenvalue whose
// neighbours are `gap` away) with p_n in FP64 and the pairs' derivative dp 2^edp of
// 2^-k T's polynomial. dp is FP32: its relative error reaches 16 eps32 ||T|| / gap
// (at most 12 of these 16 seen over disordered rings up to n = 900, 0.1 usually).
// Where the step times that is not below eps ||T|| / 2, one more evaluation and
// the secant's slope give a second step. False when the steps cannot be trusted.
__device__ __noinline__ bool last_step(const TriShared S, int n, const TriBounds B, double x, double dp, int edp, double gap,
                          double& lam) {
    double p0 = 0.0, step = 0.0;
    int e0 = 0;
    lam = x;
#pragma unroll 1
    for (int it = 0;; ++it) {
        int e;
        const double p = charpoly_value(S.d, S.e2, n, lam, e);
        if (it == 1) {
            const double den = p - scalbn(p0, max(-2000, min(2000, e0 - e)));
            if (den == 0.0) return lam == x;
            const double second = p * (lam - x) / den;
            lam -= second;
            return fabs(second) <= 0.5 * fabs(step);
        }
        p0 = p;
        e0 = e;
        step = scalbn(p / dp, max(-2000, min(2000, e - edp - S.k * (n - 1))));
        lam = x - step;
        if (!(fabs(step) <= 1e-11 * B.tnorm)) return false;
        if (fabs(step) * (32.0 * FLT_EPSILON / DBL_EPSILON) <= gap) return true;
    }
}

// One thread per eigenvalue index, FP64 result for every index: Newton in
// double-float (FP32 pairs, T rounded to them: ~1e-14 ||T||) and one last step
// with p_n in FP64 and the pairs' derivative, three FP64 operations a row
// instead of five in two or three evaluations. What is not isolated, or does
// not behave, goes to a list that the block's warps work off in FP64.
__global__ void __launch_bounds__(kEigThreads)
trieig_values_kernel(const ChainDesc* __restrict__ descs, const double* __restrict__ dd,
                     const double* __restrict__ ee, double* __restrict__ ww, int* __restrict__ status) {
    extern __shared__ double sm[];
    const ChainDesc D = descs[blockIdx.x];
    const int n = D.n;
    if ((int)(blockIdx.y * blockDim.x) >= n) return;
    TriShared S = tri_shared(sm, D.ld, true);
    double gl, gu, emax2;
    load_tridiag(D, dd, ee, S, gl, gu, emax2);
    const TriBounds B = tri_bounds(n, gl, gu, emax2);
    __shared__ float br[2 * kEigThreads];
    __shared__ int list[kEigThreads];
    __shared__ float lbr[2 * kEigThreads];
    __shared__ int cnt;
    if (threadIdx.x == 0) cnt = 0;
    const int j = blockIdx.y * blockDim.x + threadIdx.x;
    const bool active = j < n;
    if (S.d[0] != S.d[0]) {  // a chain that the reduction rejected
        if (active) ww[D.v_off + j] = NAN;
        return;
    }
    float lo = 0.f, hi = 0.f;
    block_brackets(S, n, j, active, B, lo, hi);
    double lgap, rgap;
    const double delta = bracket_slack(B);
    neighbour_gaps(br, n, j, active, lo, hi, delta, lgap, rgap);
    if (active) {
        bool done = false;
        double gap = fmin(lgap, rgap);  // beyond 2 delta the neighbours' brackets are clear of this one's
        if (!(gap > 2.0 * delta)) {
            if (isolated32(S, n, j, B, lo, hi, 64.0)) gap = 62.0 * delta;  // the first or last of a block
            else gap = isolated32(S, n, j, B, lo, hi, 2.5) ? 0.5 * delta : 0.0;
        }
        double x, dp, lam;
        int edp;
        if (gap > 0.0 && newton_df(S, n, B, lo, hi, x, dp, edp) && last_step(S, n, B, x, dp, edp, gap, lam) &&
            lam >= (double)lo - delta && lam <= (double)hi + delta) {
            ww[D.v_off + j] = lam;
            done = true;
        }
        if (!done) {
            const int q = atomicAdd(&cnt, 1);
            list[q] = j;
            lbr[2 * q] = lo;
            lbr[2 * q + 1] = hi;
        }
    }
    __syncthreads();
    list64(D, S, n, B, cnt, list, lbr, ww, status);
}

__global__ void __launch_bounds__(kEigThreads)
trieig_shift_kernel(const ChainDesc* __restrict__ descs, const double* __restrict__ dd,
                    const double* __restrict__ ee, double* __restrict__ ww, double* __restrict__ ctol,
                    int* __restrict__ status) {
    extern __shared__ double sm[];
    const ChainDesc D = descs[blockIdx.x];
    const int n = D.n;
    if ((int)(blockIdx.y * blockDim.x) >= n) return;
    TriShared S = tri_shared(sm, D.ld, false);
    __shared__ float br[2 * kEigThreads];
    __shared__ int list[kEigThreads];
    __shared__ float lbr[2 * kEigThreads];
    __shared__ int cnt;
    double gl, gu, emax2;
    load_tridiag(D, dd, ee, S, gl, gu, emax2);
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    const TriBounds B = tri_bounds(n, gl, gu, emax2);
    // the cluster tolerance of the eigenvector kernels (twisted factorisation
    // and cluster fix-up decide membership from the same number)
    if (blockIdx.y == 0 && threadIdx.x == 0) ctol[blockIdx.x] = kClusterTol * B.tnorm;
    const int j = blockIdx.y * blockDim.x + threadIdx.x;
    const bool active = j < n;
    float lo = 0.f, hi = 0.f;
    block_brackets(S, n, j, active, B, lo, hi);
    double lgap, rgap;
    const double delta = bracket_slack(B);
    neighbour_gaps(br, n, j, active, lo, hi, delta, lgap, rgap);
    if (active) {
        double x;
        if (shift_df(S.d32, S.e232, S.e2l, n, j, B, lo, hi, lgap > 2.0 * delta && rgap > 2.0 * delta, x)) {
            ww[D.v_off + j] = x;
        } else {
            const int q = atomicAdd(&cnt, 1);
            list[q] = j;
            lbr[2 * q] = lo;
            lbr[2 * q + 1] = hi;
        }
    }
    __syncthreads();
    list64(D, S, n, B, cnt, list, lbr, ww, status);  // the rest in FP64
}

}  // namespace

size_t trieig_smem_bytes(int max_ld) {
    return (size_t)max_ld * (2 * sizeof(double) + 4 * sizeof(float) + sizeof(float2));
}


cudaError_t launch_trieig_shifts(const ChainDesc* d_desc, int batch, int max_n, int max_ld, const double* d_d,
                                 const double* d_e, double* d_w, double* d_ctol, int* d_status, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    const size_t smem = trieig_smem_bytes(max_ld);
    cudaError_t err = allow_smem<trieig_shift_kernel>();
    if (err != cudaSuccess) return err;
    dim3 grid(batch, (max_n + kEigThreads - 1) / kEigThreads);
    trieig_shift_kernel<<<grid, kEigThreads, smem, st>>>(d_desc, d_d, d_e, d_w, d_ctol, d_status);
    return cudaGetLastError();
}

cudaError_t launch_trieig_values(const ChainDesc* d_desc, int batch, int max_n, int max_ld, const double* d_d,
                                 const double* d_e, double* d_w, int* d_status, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    const size_t smem = trieig_smem_bytes(max_ld);
    cudaError_t err = allow_smem<trieig_values_kernel>();
    if (err != cudaSuccess) return err;
    dim3 grid(batch, (max_n + kEigThreads - 1) / kEigThreads);
    trieig_values_kernel<<<grid, kEigThreads, smem, st>>>(d_desc, d_d, d_e, d_w, d_status);
    return cudaGetLastError();
}

}  // namespace fkg
