// vectors64.cu — FP64 eigenvectors of the tridiagonal T for the plain path's
// calc_ed(true) (src/configuration.cpp:216-219: cached_evecs, used by
// measure_ipr, measure_stiffness and measure_eigenfunctions) and for the
// FP64 free-energy gradient.
//
// Inverse iteration: for eigenvalue lambda_j, Gaussian elimination with row
// interchanges factors T - lambda_j I = P L U (U has three diagonals), and
// three solves U^{-1} L^{-1} P^T x from a fixed start vector converge to the
// eigenvector. Eigenvalues closer than 1e-5 ||T|| form a cluster: one thread
// computes the cluster's vectors in order and orthogonalises each iterate
// against the cluster's earlier vectors (modified Gram-Schmidt), so exactly
// degenerate eigenvalues (the U = 0 lattices) still get an orthonormal basis.
// Vectors outside a cluster are orthogonal to about eps ||T|| / gap < 1e-11.
// Output row-major Z[i*ld + j] = component i of eigenvector j.
#include <cfloat>

#include "fkg_common.cuh"

namespace fkg {
namespace {

struct LU {
    double* r0;   // reciprocals of the diagonal of U
    double* u1;   // first superdiagonal of U
    double* u2;   // second superdiagonal of U (fill-in from interchanges)
    double* m;    // multipliers of L
    int* piv;     // 1 where rows i and i+1 were interchanged
};

// |x| as an integer: comparisons of FP64 numbers off the FP64 pipe
__device__ __forceinline__ long long abs_bits(double x) { return __double_as_longlong(x) & 0x7fffffffffffffffll; }

// The pivots are kept as reciprocals: one FP64 division per elimination step
// serves the multiplier and the three back substitutions, which then only
// multiply (a division is a long dependent sequence on the FP64 pipe; the
// solves are chains of n dependent steps). A pivot below pivmin is replaced by
// +-pivmin before its reciprocal is taken.
__device__ void factor(const double* d, const double* e, int n, double lam, double pivmin, LU f) {
    const long long pivbits = abs_bits(pivmin);
    auto guard = [&](double x) { return abs_bits(x) < pivbits ? (x < 0.0 ? -pivmin : pivmin) : x; };
    double cd = d[0] - lam, cs = n > 1 ? e[0] : 0.0;  // active row: diagonal and superdiagonal
    for (int i = 0; i + 1 < n; ++i) {
        const double sub = e[i], an = d[i + 1] - lam, en = i + 2 < n ? e[i + 1] : 0.0;
        if (abs_bits(cd) >= abs_bits(sub)) {
            const double r = 1.0 / guard(cd), mu = sub * r;
            f.r0[i] = r; f.u1[i] = cs; f.u2[i] = 0.0; f.m[i] = mu; f.piv[i] = 0;
            cd = an - mu * cs;
            cs = en;
        } else {
            const double r = 1.0 / guard(sub), mu = cd * r;
            f.r0[i] = r; f.u1[i] = an; f.u2[i] = en; f.m[i] = mu; f.piv[i] = 1;
            cd = cs - mu * an;
            cs = -mu * en;
        }
    }
    f.r0[n - 1] = 1.0 / guard(cd);
}

// x <- (P L U)^{-1} x, in place. The recurrences run in registers, with the rows
// of the next four steps loaded ahead.
__device__ void solve(LU f, int n, double* x) {
    double cur = x[0];
    if (n > 1) {
        double nm[4], nx[4];
        int np[4];
        auto fetch = [&](int i0) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int i = min(i0 + u, n - 2);
                nm[u] = f.m[i]; np[u] = f.piv[i]; nx[u] = x[i + 1];
            }
        };
        fetch(0);
        for (int i0 = 0; i0 + 1 < n; i0 += 4) {
            double tm[4], tx[4];
            int tp[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) { tm[u] = nm[u]; tp[u] = np[u]; tx[u] = nx[u]; }
            if (i0 + 5 < n) fetch(i0 + 4);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (i0 + u + 1 < n) {
                    const double y = tp[u] ? tx[u] : cur, z = tp[u] ? cur : tx[u];
                    x[i0 + u] = y;
                    cur = z - tm[u] * y;
                }
        }
    }
    double x1 = cur * f.r0[n - 1], x2 = 0.0;
    x[n - 1] = x1;
    if (n < 2) return;
    {
        const double t = (x[n - 2] - f.u1[n - 2] * x1) * f.r0[n - 2];
        x2 = x1;
        x1 = t;
        x[n - 2] = t;
    }
    if (n < 3) return;
    double c0[4], c1[4], c2[4], cr[4];
    auto fetch = [&](int i0) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = max(i0 - u, 0);
            c0[u] = x[i]; c1[u] = f.u1[i]; c2[u] = f.u2[i]; cr[u] = f.r0[i];
        }
    };
    fetch(n - 3);
    for (int i0 = n - 3; i0 >= 0; i0 -= 4) {
        double t0[4], t1[4], t2[4], tr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) { t0[u] = c0[u]; t1[u] = c1[u]; t2[u] = c2[u]; tr[u] = cr[u]; }
        if (i0 >= 4) fetch(i0 - 4);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 >= u) {
                const double t = (t0[u] - t1[u] * x1 - t2[u] * x2) * tr[u];
                x2 = x1;
                x1 = t;
                x[i0 - u] = t;
            }
    }
}

// x 2^-k by its exponent field; subnormal numbers, before or after, become 0
__device__ __forceinline__ double scale_down(double x, int k) {
    const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
    return e == 0 || e <= k ? 0.0 : __hiloint2double(hi - k * (1 << 20), __double2loint(x));
}

// One thread per vector, a warp per CTA: the recurrences are serial, and a warp's FP64 instruction takes 64-76
// cycles of its scheduler whatever its latency, so what counts is their number: 29 a row for the factorisation and
// the three solves. The start vector comes from 32 sines by angle addition, the first forward elimination runs
// inside the factorisation, reciprocals take the hardware's approximation and one third-order step, comparisons and
// the scaling between solves (by powers of two) are integer work. Rows are stored [i][vector] (coalesced) and read
// four ahead.
// A cluster's members follow one another on the lane that leads it; their orthogonalisation is the whole warp's.
// Measured (one thread's rows apart, branches, divisions and sines before): 32 chains of N = 225 1.41 -> 0.45 ms,
// 256 of N = 576 27.4 -> 6.0 ms, one of N = 64 0.31 -> 0.11 ms; clusters of 4, 8 and 30 (64 chains of N = 256 without f)
// 57 -> 17 ms, 54 with the leading lane orthogonalising.
__global__ void __launch_bounds__(32, 16)  // 12 CTAs an SM (168 registers): 7.3 ms
stein_kernel(const ChainDesc* __restrict__ descs, const double* __restrict__ dd, const double* __restrict__ ee,
             const double* __restrict__ ww, double* __restrict__ Zws, double* __restrict__ scratch) {
    extern __shared__ double2 de[];  // d_i, e_i
    __shared__ double2 rot[32];      // sin, cos of 0.7 i
    const ChainDesc D = descs[blockIdx.x];
    const int n = D.n, ld = D.ld, lane = threadIdx.x, j = blockIdx.y * 32 + lane;
    if ((int)blockIdx.y * 32 >= n) return;
    for (int i = lane; i < n; i += 32) de[i] = make_double2(dd[D.v_off + i], i + 1 < n ? ee[D.v_off + i] : 0.0);
    sincos(0.7 * lane, &rot[lane].x, &rot[lane].y);
    __syncwarp();
    double gl = DBL_MAX, gu = -DBL_MAX;
    for (int i = lane; i < n; i += 32) {
        const double r = (i > 0 ? fabs(de[i - 1].y) : 0.0) + fabs(de[i].y);
        gl = fmin(gl, de[i].x - r);
        gu = fmax(gu, de[i].x + r);
    }
    const double tnorm = fmax(fabs(warp_min(gl)), fabs(warp_max(gu)));
    const double ortol = 1e-5 * tnorm, pivmin = DBL_EPSILON * tnorm + DBL_MIN;
    const double* w = ww + D.v_off;
    int members = 0;  // of the cluster that this lane leads
    if (j < n && !(j > 0 && w[j] - w[j - 1] <= ortol))
        for (members = 1; j + members < n && w[j + members] - w[j + members - 1] <= ortol;) ++members;
    double* Z = Zws + D.a_off;
    // chain c owns [6 a_off_c, 6 a_off_c + 6 ld_c^2): planes of ld x ld, this thread's column j
    const size_t plane = (size_t)ld * ld;
    double* const r0 = scratch + 6 * (size_t)D.a_off + j;  // reciprocals of the diagonal of U
    double* const u1 = r0 + plane;                         // its superdiagonals
    double* const u2 = u1 + plane;
    double* const ml = u2 + plane;                         // multipliers of L
    double* const yy = ml + plane;                         // forward solution
    unsigned* const pv = reinterpret_cast<unsigned*>(yy + plane - j) + j;  // row interchanges, 32 rows a word
    const long long pivbits = abs_bits(pivmin);
    auto guard = [&](double x) { return abs_bits(x) < pivbits ? copysign(pivmin, x) : x; };
    const double rs = sin(0.7 * 32), rc = cos(0.7 * 32);
    for (int r = 0; __any_sync(0xffffffffu, r < members); ++r) {
        const bool on = r < members;
        const int jj = j + r;
        double* const z = Z + jj;
        double cur, rl;
        unsigned bits = 0;
        if (on) {
            // a perturbation of 2 eps ||T|| keeps identical eigenvalues of a cluster apart
            const double lam = w[jj] + r * 2.0 * DBL_EPSILON * tnorm;
            // fixed start vector 1 + sin(0.7 i + 1.3 jj) / 4: ps, pc the sine and cosine at the last multiple of 32
            double ps, pc;
            sincos(1.3 * jj, &ps, &pc);
            ps *= 0.25;
            pc *= 0.25;
            auto start = [&](int i) {
                if ((i & 31) == 0 && i > 0) {
                    const double t = fma(ps, rc, pc * rs);
                    pc = fma(pc, rc, -ps * rs);
                    ps = t;
                }
                const double2 q = rot[i & 31];
                return fma(pc, q.x, fma(ps, q.y, 1.0));
            };
            // factorisation, with the first forward elimination
            double cd = de[0].x - lam, cs = de[0].y;  // active row: diagonal, superdiagonal, right side (cur)
            cur = start(0);
            for (int i = 0; i + 1 < n; ++i) {
                const double sub = de[i].y, an = de[i + 1].x - lam, en = de[i + 1].y, nx = start(i + 1);
                const bool swap = abs_bits(cd) < abs_bits(sub);
                const double rp = recip64(guard(swap ? sub : cd)), mu = (swap ? cd : sub) * rp;
                const double a1 = swap ? an : cs, a2 = swap ? en : 0.0, y = swap ? nx : cur;
                const size_t o = (size_t)i * ld;
                r0[o] = rp;
                u1[o] = a1;
                u2[o] = a2;
                ml[o] = mu;
                yy[o] = y;
                bits |= (unsigned)swap << (i & 31);
                if ((i & 31) == 31) {
                    pv[(size_t)(i >> 5) * ld] = bits;
                    bits = 0;
                }
                cur = fma(-mu, y, swap ? cur : nx);
                cd = fma(-mu, a1, swap ? cs : an);
                cs = fma(-mu, a2, swap ? 0.0 : en);
            }
            if ((n - 1) & 31) pv[(size_t)((n - 1) >> 5) * ld] = bits;
            rl = recip64(guard(cd));
        }
        double nrm, sg;  // squared norm, a component with the vector's sign
        long long best;  // the largest component (the first of equal ones)
        for (int it = 0;; ++it) {
            if (on) {
                // back substitution
                double x1 = cur * rl, x2 = 0.0;
                best = abs_bits(x1);
                sg = x1;
                double sq[4] = {x1 * x1, 0.0, 0.0, 0.0};  // four sums round less than one
                z[(size_t)(n - 1) * ld] = x1;
                double cy[4], c1[4], c2[4], cr[4];
                auto fetch = [&](int i0) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const size_t o = (size_t)max(i0 - u, 0) * ld;
                        cy[u] = yy[o]; c1[u] = u1[o]; c2[u] = u2[o]; cr[u] = r0[o];
                    }
                };
                if (n > 1) fetch(n - 2);
                for (int i0 = n - 2; i0 >= 0; i0 -= 4) {
                    double ty[4], t1[4], t2[4], tr[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) { ty[u] = cy[u]; t1[u] = c1[u]; t2[u] = c2[u]; tr[u] = cr[u]; }
                    if (i0 >= 4) fetch(i0 - 4);
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i0 >= u) {
                            const double x = fma(-t1[u], x1, fma(-t2[u], x2, ty[u])) * tr[u];
                            x2 = x1;
                            x1 = x;
                            z[(size_t)(i0 - u) * ld] = x;
                            const long long ab = abs_bits(x);
                            if (ab >= best) { best = ab; sg = x; }
                            if (it == 2) sq[u] = fma(x, x, sq[u]);
                        }
                }
                nrm = (sq[0] + sq[1]) + (sq[2] + sq[3]);
            }
            if (r > 0) {
                // orthogonalise against the cluster's earlier vectors, the whole warp on one vector after the other
                // (a lane that works alone takes as much of the FP64 pipe as 32), a lane's rows lane + 32 q
                __syncwarp();
                for (unsigned todo = __ballot_sync(0xffffffffu, on); todo; todo &= todo - 1) {
                    const int l = __ffs(todo) - 1, first = j - lane + l;
                    double* const x = Z + first + r;
                    for (int q = first; q < first + r; ++q) {
                        double dot = 0.0;
                        for (int i = lane; i < n; i += 32) dot = fma(Z[(size_t)i * ld + q], x[(size_t)i * ld], dot);
                        dot = warp_sum(dot);
                        for (int i = lane; i < n; i += 32) x[(size_t)i * ld] -= dot * Z[(size_t)i * ld + q];
                    }
                    long long top = -1;
                    double tx = 0.0, sum = 0.0;
                    int ti = n;
                    for (int i = lane; i < n; i += 32) {
                        const double y = x[(size_t)i * ld];
                        if (abs_bits(y) > top) { top = abs_bits(y); tx = y; ti = i; }
                        sum = fma(y, y, sum);
                    }
                    sum = warp_sum(sum);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        const long long ot = __shfl_xor_sync(0xffffffffu, top, o);
                        const double ox = __shfl_xor_sync(0xffffffffu, tx, o);
                        const int oi = __shfl_xor_sync(0xffffffffu, ti, o);
                        if (ot > top || (ot == top && oi < ti)) { top = ot; tx = ox; ti = oi; }
                    }
                    if (lane == l) { best = top; sg = tx; nrm = sum; }
                }
                __syncwarp();
            }
            if (on) {
                const int k = (int)(best >> 52) - 1023;  // 1024: not a number, which stays so
                if (it == 2) {
                    if (!(nrm > 1e-280 && nrm < 1e280) && k < 1024) {  // squares out of range: the scaled vector
                        nrm = 0.0;
                        for (int i = 0; i < n; ++i) {
                            const double x = scale_down(z[(size_t)i * ld], k);
                            z[(size_t)i * ld] = x;
                            nrm = fma(x, x, nrm);
                        }
                    }
                } else {
                    // scaled forward elimination
                    const double nan = k == 1024 ? (double)NAN : 0.0;
                    cur = scale_down(z[0], k) + nan;
                    double cz[4], cm[4];
                    auto fetch2 = [&](int i0) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const size_t o = (size_t)min(i0 + u, n - 2) * ld;
                            cm[u] = ml[o];
                            cz[u] = z[o + ld];
                        }
                    };
                    if (n > 1) fetch2(0);
                    for (int i0 = 0; i0 + 1 < n; i0 += 4) {
                        double tm[4], tz[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) { tm[u] = cm[u]; tz[u] = cz[u]; }
                        if (i0 + 5 < n) fetch2(i0 + 4);
                        if ((i0 & 31) == 0) bits = pv[(size_t)(i0 >> 5) * ld];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (i0 + u + 1 < n) {
                                const bool swap = bits >> ((i0 + u) & 31) & 1;
                                const double nx = scale_down(tz[u], k), y = swap ? nx : cur;
                                yy[(size_t)(i0 + u) * ld] = y;
                                cur = fma(-tm[u], y, swap ? cur : nx);
                            }
                    }
                }
            }
            if (it == 2) break;
        }
        // sign: largest component positive (deterministic output)
        if (on) {
            const double sc = copysign(1.0 / sqrt(nrm), sg);
#pragma unroll 4
            for (int i = 0; i < n; ++i) z[(size_t)i * ld] *= sc;
        }
    }
}

// Mixed path: the twisted-factorisation vectors are accurate for isolated
// eigenvalues but may coincide inside clusters of (nearly) equal eigenvalues
// (gaps <= 1e-5 ||T||; the twisted factorisation skips those members, and
// this kernel runs beside it on a second stream). One CTA per chain computes
// the clusters' vectors by FP64 inverse iteration, the members of several
// clusters at once: thread g
// owns member g (its LU factors and iterate in the chain's scratch, 6 ld
// doubles), and after each of the three solves one warp per cluster
// orthonormalises the cluster's iterates in order (modified Gram-Schmidt,
// lanes over the rows). A wave holds at most min(256, ld / 6) members; a
// longer cluster is done in chunks, each chunk's iterates first made
// orthogonal to the cluster's vectors finished in earlier waves. Chains
// without a cluster leave after the scan.
constexpr int kCfThreads = 256;

__global__ void __launch_bounds__(kCfThreads)
cluster_fix_kernel(const ChainDesc* __restrict__ descs, const double* __restrict__ dd, const double* __restrict__ ee,
                   const double* __restrict__ ww, const double* __restrict__ ctol, float* __restrict__ Zws,
                   float* __restrict__ zscale, double* __restrict__ scratch) {
    extern __shared__ double smc[];
    const ChainDesc D = descs[blockIdx.x];
    const int n = D.n, ld = D.ld;
    double* d = smc;
    double* e = d + ld;
    double* w = e + ld;
    __shared__ int sj[kCfThreads], sr[kCfThreads], cls[kCfThreads + 1], cfin[kCfThreads];
    __shared__ int s_nslots, s_ncl, s_pos, s_cstart, s_cend;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < n; i += blockDim.x) {
        d[i] = dd[D.v_off + i];
        e[i] = i + 1 < n ? ee[D.v_off + i] : 0.0;
        w[i] = ww[D.v_off + i];
    }
    __syncthreads();
    // the tolerance the shift kernel recorded (the twisted factorisation skips
    // exactly these members)
    const double ortol = ctol[blockIdx.x], tnorm = ortol / kClusterTol;
    const double pivmin = DBL_EPSILON * tnorm + DBL_MIN;
    __shared__ unsigned close[32];  // bit i: member i belongs to the cluster of i - 1
    int any = 0;
    for (int i = tid; i < (n + 31) / 32 * 32; i += blockDim.x) {
        const bool c = i > 0 && i < n && w[i] - w[i - 1] <= ortol;
        const unsigned b = __ballot_sync(0xffffffffu, c);
        if (lane == 0) close[i >> 5] = b;
        any |= c;
    }
    if (!__syncthreads_or(any)) return;
    auto joined = [&](int i) { return close[i >> 5] >> (i & 31) & 1; };
    float* Z = Zws + D.a_off;
    double* base0 = scratch + D.a_off;  // ld * ld doubles of this chain
    const int cap = min(kCfThreads, ld / 6);
    if (tid == 0) { s_pos = 0; s_cstart = 0; s_cend = 0; }
    __syncthreads();
    for (;;) {
        // ---- the next wave (thread 0 walks the spectrum): whole clusters, or
        //      a chunk of one that does not fit; cfin[c] = the cluster's first
        //      member, members cfin[c] .. sj[cls[c]] - 1 are finished ----
        if (tid == 0) {
            int pos = s_pos, cstart = s_cstart, cend = s_cend, g = 0, c = 0;
            while (pos < n && g < cap) {
                if (pos >= cend) {  // at a cluster boundary: find the next cluster
                    int end = pos + 1;
                    while (end < n && joined(end)) ++end;
                    if (end - pos < 2) { pos = end; continue; }
                    cstart = pos;
                    cend = end;
                }
                const int take = min(cend - pos, cap - g);
                cls[c] = g;
                cfin[c] = cstart;
                ++c;
                for (int q = 0; q < take; ++q) { sj[g + q] = pos + q; sr[g + q] = pos + q - cstart; }
                g += take;
                pos += take;
            }
            cls[c] = g;
            s_nslots = g;
            s_ncl = c;
            s_pos = pos;
            s_cstart = cstart;
            s_cend = cend;
        }
        __syncthreads();
        const int nslots = s_nslots, ncl = s_ncl;
        if (nslots == 0) break;
        double* base = base0 + (size_t)min(tid, cap - 1) * 6 * ld;
        LU f{base, base + ld, base + 2 * ld, base + 3 * ld, reinterpret_cast<int*>(base + 4 * ld)};
        double* x = base + 5 * ld;
        if (tid < nslots) {
            const int jj = sj[tid];
            // a perturbation of 2 eps ||T|| per rank keeps identical eigenvalues apart
            const double lam = w[jj] + sr[tid] * 2.0 * DBL_EPSILON * tnorm;
            factor(d, e, n, lam, pivmin, f);
        }
        // fixed start vectors, by the warps that factor nothing (nslots <= ld / 6 leaves some): a sine costs
        // as much as a row's division, and a member's thread would evaluate n of them in turn
        const int nf = (nslots + 31) / 32 * 32;
        for (int q = tid - nf; q >= 0 && q < nslots * n; q += kCfThreads - nf) {
            const int g = q / n, i = q - g * n, jj = sj[g];
            base0[(size_t)g * 6 * ld + 5 * ld + i] = 1.0 + 0.25 * sin(0.7 * i + 1.3 * jj);
        }
        __syncthreads();
        for (int it = 0; it < 3; ++it) {
            if (tid < nslots) solve(f, n, x);
            __syncthreads();
            for (int c = warp; c < ncl; c += kCfThreads / 32) {
                const int g0 = cls[c], k = cls[c + 1] - g0;
                for (int f = cfin[c]; f < sj[g0]; ++f) {  // the cluster's vectors from earlier waves
                    for (int m = 0; m < k; ++m) {
                        double* xm = base0 + (size_t)(g0 + m) * 6 * ld + 5 * ld;
                        double dp = 0.0;
                        for (int i = lane; i < n; i += 32) dp += (double)Z[(size_t)i * ld + f] * xm[i];
                        const double dot = warp_sum(dp);
                        for (int i = lane; i < n; i += 32) xm[i] -= dot * (double)Z[(size_t)i * ld + f];
                        __syncwarp();
                    }
                }
                for (int q = 0; q < k; ++q) {
                    double* xq = base0 + (size_t)(g0 + q) * 6 * ld + 5 * ld;
                    double part = 0.0;
                    for (int i = lane; i < n; i += 32) part += xq[i] * xq[i];
                    const double sc = 1.0 / sqrt(warp_sum(part));
                    for (int i = lane; i < n; i += 32) xq[i] *= sc;
                    __syncwarp();
                    for (int m = q + 1; m < k; ++m) {
                        double* xm = base0 + (size_t)(g0 + m) * 6 * ld + 5 * ld;
                        double dp = 0.0;
                        for (int i = lane; i < n; i += 32) dp += xq[i] * xm[i];
                        const double dot = warp_sum(dp);
                        for (int i = lane; i < n; i += 32) xm[i] -= dot * xq[i];
                        __syncwarp();
                    }
                }
            }
            __syncthreads();
        }
        for (int g = warp; g < nslots; g += kCfThreads / 32) {
            const double* xg = base0 + (size_t)g * 6 * ld + 5 * ld;
            const int jj = sj[g];
            for (int i = lane; i < n; i += 32) Z[(size_t)i * ld + jj] = (float)xg[i];
            if (lane == 0) zscale[D.v_off + jj] = 1.f;  // written normalised
        }
        __syncthreads();
    }
}

}  // namespace

cudaError_t launch_cluster_fix_f32(const ChainDesc* d_desc, int batch, int max_ld, const double* d_d,
                                   const double* d_e, const double* d_w, const double* d_ctol, float* d_Z,
                                   float* d_zscale, double* d_scratch, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    const size_t smem = sizeof(double) * 3 * (size_t)max_ld;
    cudaError_t err = allow_smem<cluster_fix_kernel>();
    if (err != cudaSuccess) return err;
    cluster_fix_kernel<<<batch, kCfThreads, smem, st>>>(d_desc, d_d, d_e, d_w, d_ctol, d_Z, d_zscale,
                                                         d_scratch);
    return cudaGetLastError();
}

size_t stein_scratch_elems(long long a_total) { return (size_t)6 * a_total; }

cudaError_t launch_stein_f64(const ChainDesc* d_desc, int batch, int max_n, int max_ld, const double* d_d,
                             const double* d_e, const double* d_w, double* d_Z, double* d_scratch, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    stein_kernel<<<dim3(batch, (max_n + 31) / 32), 32, sizeof(double2) * max_ld, st>>>(d_desc, d_d, d_e, d_w, d_Z,
                                                                                        d_scratch);
    return cudaGetLastError();
}

}  // namespace fkg
