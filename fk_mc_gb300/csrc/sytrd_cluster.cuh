// sytrd_cluster.cuh — Householder tridiagonalisation by a thread-block cluster
// per chain, the trailing matrix held in the cluster's shared memory.
//
// Replaces the first half of Eigen::SelfAdjointEigenSolver at
// src/configuration.cpp:213; the Hamiltonian build (src/configuration.cpp:79-91)
// and the dense copy (:212) are fused into the tile fill.
//
// Algorithm (panel of NB reflectors, deferred symmetric rank-2k update), as in
// LAPACK's dlatrd: per column the pending updates of the panel on that column, the
// reflector, p = A22 v with the stale trailing matrix corrected by the panel's
// V and W; after the panel A22 -= V W^T + W V^T.
//
// Arithmetic (template parameter P):
//   F32  FP32 throughout (the mixed path's reduction; sytrd_f32.cu);
//   Fix  FP64-grade arithmetic on the integer pipe (sytrd_f64.cu). GB300 issues one FP64
//        multiply-add per warp every 64-76 cycles of a sub-partition, one
//        32 x 32 -> 64 bit integer multiplication every 4 (measured). All matrix
//        and vector entries are 64-bit fixed-point numbers relative to S, the
//        power of two above the largest row sum of |H| (so ||H||_2 <= S), held as
//        two limbs x = hi 2^LO + lo (hi 32 bits, |lo| <= 2^(LO - 1); formats at
//        struct Fix). A product is three integer multiplications: hi hi into one
//        64-bit sum, hi lo + lo hi into another; lo lo is dropped. The sums are
//        exact: the results are bounded by the norms (|A v| <= sqrt(2) S, |w| <=
//        2 S, the cross sums by sqrt(n) times the limbs' ranges), and
//        intermediate wrap-around modulo 2^64 is harmless. Where a partial sum leaves
//        its lane its cross sum is rounded to the other's unit, so a result's last bits
//        depend on how many warps and CTAs share the chain (but not on their timing).
//        Orthogonal
//        transformations keep ||A||_2, so no entry outgrows its format. The
//        rounding is half a quantum per entry and panel where FP64 rounds every
//        product; the norm of a column is an exact integer sum,
//        its inverse square root a Newton iteration from the FP32 estimate on
//        64-bit integers (the FP64 square root and divisions cost ~1100 cycles
//        each per column). Errors against 34-digit arithmetic
//        (rms over the spectrum / ||H||; FP64 kernel before, this): N = 64 6.0e-17,
//        2.6e-17; N = 64 with U = 20 2.1e-16, 4.2e-17; N = 125 5.1e-17, 2.5e-17; N = 144
//        5.3e-17, 3.8e-17; N = 196 7.0e-17, 3.8e-17.
//
// Work split. A chain's lower 32 x 32 tiles are numbered by decreasing tile
// column, so the tiles alive at a step are always a prefix; tile t belongs to
// CTA t mod C and the tiles that die first are the ones kept in global memory
// when shared memory is too small. Inside a tile lane (g, t4) owns rows g + 8 m
// and columns 8 q + 2 t4 + {0, 1}, stored as 16-byte units in lane order (every
// access conflict free). A matrix-vector product reads a tile once, uses each
// entry for its row and its column sum and reduces with shuffles; a warp takes
// consecutive tiles, which share their column sums.
// Two cluster barriers per column: after the column and its norm have been
// written to every CTA's shared memory, and after the partial products have;
// the rest of a column is computed redundantly by every CTA.
#pragma once
#include <cooperative_groups.h>

#include <cfloat>

#include "fkg_common.cuh"

namespace cg = cooperative_groups;

namespace fkg {
namespace {

constexpr int kTileElems = kTile * kTile;
constexpr int kMaxTileRows = 32;  // n <= 1024
typedef long long ll;
typedef unsigned long long ull;

// 64-bit warp sum in three 32-bit reductions
__device__ __forceinline__ ll warp_sum_ll(ll x) {
    const unsigned a = (unsigned)x & 0x3fffffu, b = (unsigned)((ull)x >> 22) & 0x3fffffu;
    const int c = (int)(x >> 44);
    const ull sa = __reduce_add_sync(0xffffffffu, a), sb = __reduce_add_sync(0xffffffffu, b);
    const ull sc = (ull)(ll)__reduce_add_sync(0xffffffffu, c);
    return (ll)(sa + (sb << 22) + (sc << 44));
}

__device__ __forceinline__ float add_mod(float a, float b) { return a + b; }
__device__ __forceinline__ ll add_mod(ll a, ll b) { return (ll)((ull)a + (ull)b); }

// Sums of VN values over the lanes that differ in the lane bits `HI`, `HI`/2,
// ... (VN of them halve), by recursive halving. After it the lane holds the total of
// value `idx` over those lanes.
template <int VN, int HI, typename T>
__device__ __forceinline__ T reduce_scatter(T (&x)[VN], int lane, int& idx) {
    int base = 0;
#pragma unroll
    for (int half = VN / 2, o = HI; half >= 1; half >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int m = 0; m < half; ++m) {
            const T send = up ? x[m] : x[m + half];
            const T keep = up ? x[m + half] : x[m];
            x[m] = add_mod(keep, __shfl_xor_sync(0xffffffffu, send, o));
        }
        if (up) base += half;
    }
    idx = base;
    return x[0];
}

// time of a column in k cycles, see launch_cluster: base, per row, per tile of a CTA's mean share and per tile of it in
// global memory, for a cluster's barriers and for each CTA beyond the first; its relative increase for each further CTA
// on an SM
struct ColumnCost {
    double base, row, tile, spill, cluster, cta, shared;
};

// W warps a CTA; four CTAs of 4 warps, two of 8 or one of 16 share an SM
template <int W>
struct F32 {
    static constexpr int kWarps = W, kOcc = 16 / W;
    static constexpr ColumnCost kCost = W == 4   ? ColumnCost{3.99, 0.0, 0.398, 0.0, 1.25, 0.214, 0.15}
                                        : W == 8 ? ColumnCost{4.72, 0.00248, 0.080, 0.095, 0.70, 0.139, 0.15}
                                                 : ColumnCost{5.23, 0.00152, 0.095, 0.041, 0.93, 0.166, 0.15};
    using V = float;  // matrix / vector entry
    using S = float;  // sum
    using G = float;  // reflectors in global memory
    static constexpr int kPwWords = kWarps;  // per-warp copies of the product
    struct Acc {
        float s;
    };
    static __device__ __forceinline__ void zero(Acc& a) { a.s = 0.f; }
    static __device__ __forceinline__ void mac(Acc& a, V x, V y) { a.s = fmaf(x, y, a.s); }
    static __device__ __forceinline__ void mac2(Acc& a, V x0, V y0, V x1, V y1) { a.s = fmaf(x1, y1, fmaf(x0, y0, a.s)); }
    static __device__ __forceinline__ S sum(const Acc& a) { return a.s; }
    static __device__ __forceinline__ V vzero() { return 0.f; }
    static __device__ __forceinline__ void ld4(const void* t, int q, int lane, V (&a)[4]) {
        const float4 x = ((const float4*)t)[q * 32 + lane];
        a[0] = x.x; a[1] = x.y; a[2] = x.z; a[3] = x.w;
    }
    static __device__ __forceinline__ void st4(void* t, int q, int lane, const V (&a)[4]) {
        ((float4*)t)[q * 32 + lane] = make_float4(a[0], a[1], a[2], a[3]);
    }
    static __device__ __forceinline__ void ld2(const V* p, V (&a)[2]) {
        const float2 x = *(const float2*)p;
        a[0] = x.x; a[1] = x.y;
    }
    static __device__ __forceinline__ V get(const void* t, int off) { return ((const float*)t)[off]; }
    static __device__ __forceinline__ void put(void* t, int off, V v) { ((float*)t)[off] = v; }
    static __device__ __forceinline__ V upd(V a, const Acc& u) { return a - u.s; }  // a - u (rank-2k update)
};

// LO: bits of the low limb (quanta 2^-(30 + LO) S of a matrix, 2^-(30 + LO) of
// v, 2^-(29 + LO) S of w). 27 keeps the cross sums below 2^63 for n <= 1024, 28 for
// n <= 256. W warps a CTA; two CTAs of 4 warps or one of 8 (~240 registers a
// thread) share an SM.
template <int LO, int W>
struct Fix {
    static constexpr int kWarps = W, kOcc = 8 / W;
    static constexpr ColumnCost kCost = {8.8, 0.0034, 0.68, 0.0, 0.8, 0.0, 0.0};
    static constexpr int kLo = LO;
    using V = int2;  // (hi, lo)
    using S = ll;
    using G = double;
    static constexpr int kPwWords = 3;  // 21-bit limbs of the product, one copy
    struct Acc {
        ull h, x;
    };
    static __device__ __forceinline__ void zero(Acc& a) { a.h = a.x = 0; }
    static __device__ __forceinline__ ull mw(int a, int b) {
        ull r;
        asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
        return r;
    }
    static __device__ __forceinline__ void mac(Acc& a, V p, V q) {
        a.h += mw(p.x, q.x);
        a.x += mw(p.x, q.y) + mw(p.y, q.x);
    }
    // two products at a time: one three-input 64-bit addition takes two of them
    static __device__ __forceinline__ void mac2(Acc& a, V p0, V q0, V p1, V q1) {
        a.h += mw(p0.x, q0.x) + mw(p1.x, q1.x);
        a.x += mw(p0.x, q0.y) + mw(p0.y, q0.x);
        a.x += mw(p1.x, q1.y) + mw(p1.y, q1.x);
    }
    // the sum in units of the hi hi products
    static __device__ __forceinline__ S sum(const Acc& a) {
        return (ll)(a.h + (ull)(((ll)a.x + (1 << (LO - 1))) >> LO));
    }
    static __device__ __forceinline__ V vzero() { return make_int2(0, 0); }
    static __device__ __forceinline__ V split(ll a) {
        const int lo = ((int)a << (32 - LO)) >> (32 - LO);
        return make_int2((int)((a - lo) >> LO), lo);
    }
    static __device__ __forceinline__ ll join(V v) { return (ll)v.x * (1 << LO) + v.y; }
    // x rounded from units 2^-XB to units 2^-YB
    template <int XB, int YB>
    static __device__ __forceinline__ ll round_to(ll x) {
        if constexpr (XB > YB) return (x + (1ll << (XB - YB - 1))) >> (XB - YB);
        else return x << (YB - XB);
    }
    static __device__ __forceinline__ void ld4(const void* t, int q, int lane, V (&a)[4]) {
        const int4 h = ((const int4*)t)[q * 32 + lane], l = ((const int4*)t)[256 + q * 32 + lane];
        a[0] = make_int2(h.x, l.x); a[1] = make_int2(h.y, l.y);
        a[2] = make_int2(h.z, l.z); a[3] = make_int2(h.w, l.w);
    }
    static __device__ __forceinline__ void st4(void* t, int q, int lane, const V (&a)[4]) {
        ((int4*)t)[q * 32 + lane] = make_int4(a[0].x, a[1].x, a[2].x, a[3].x);
        ((int4*)t)[256 + q * 32 + lane] = make_int4(a[0].y, a[1].y, a[2].y, a[3].y);
    }
    static __device__ __forceinline__ void ld2(const V* p, V (&a)[2]) {
        const int4 x = *(const int4*)p;
        a[0] = make_int2(x.x, x.y); a[1] = make_int2(x.z, x.w);
    }
    static __device__ __forceinline__ V get(const void* t, int off) {
        return make_int2(((const int*)t)[off], ((const int*)t)[kTileElems + off]);
    }
    static __device__ __forceinline__ void put(void* t, int off, V v) {
        ((int*)t)[off] = v.x;
        ((int*)t)[kTileElems + off] = v.y;
    }
    // a - u: u = sum of v w products in units 2^-59 S, a in 2^-(30 + LO) S. Rounded
    // with all the bits of the cross products: from the sum in whole units every
    // second to eighth rounding would be a tie, whose common direction adds up over
    // the entries and columns.
    static __device__ __forceinline__ ll upd_ll(V a, const Acc& u) {
        constexpr int sh = 29 - LO;
        const ll low = ((ll)((unsigned)u.h & ((1u << sh) - 1)) << LO) + (ll)u.x + (1 << 28);
        return join(a) - (((ll)u.h >> sh) + (low >> 29));
    }
    static __device__ __forceinline__ V upd(V a, const Acc& u) { return split(upd_ll(a, u)); }
    // w = tau p - K v: p in units 2^-60 S, K v (kv) in 2^-59 S
    static __device__ __forceinline__ V w_entry(ll p, ll tau, const Acc& kv) {
        const ll k60 = (ll)(2 * kv.h) + (((ll)kv.x + (1 << (LO - 2))) >> (LO - 1));
        return split(round_to<60, 29 + LO>(__mul64hi(p * 4, tau) - k60));
    }
    // K = tau^2 p.v / 2 (p.v in units 2^-60 S)
    static __device__ __forceinline__ V k_value(ll pv, ll tau) {
        return split(round_to<60, 29 + LO>(__mul64hi(__mul64hi(pv * 2, tau) * 4, tau)));
    }
};

// the NB entries of one row of Vp or Wp, in 16-byte loads
template <int NB, typename V>
__device__ __forceinline__ void ld_row(const V* p, V (&r)[NB]) {
    constexpr int kPer = 16 / sizeof(V);
    static_assert(NB % kPer == 0, "rows of whole 16-byte units");
#pragma unroll
    for (int q = 0; q < NB / kPer; ++q) {
        const int4 x = ((const int4*)p)[q];
        memcpy(&r[q * kPer], &x, 16);
    }
}

// offset of entry (r, c) of a tile (lane-owned 16-byte units)
__device__ __forceinline__ int elem_off(int r, int c) {
    const int q = ((r >> 4) & 1) * 4 + (c >> 3), lane = (r & 7) * 4 + ((c & 7) >> 1);
    return (q * 32 + lane) * 4 + ((r >> 3) & 1) * 2 + (c & 1);
}

// Reflector scalars of the fixed-point path. x: the column (integers, quantum
// q), s2 = sum x_i^2 over the column, alpha its first entry; all values relative
// to 2^(64 - z/2), z an even shift that normalises s2: xn = sqrt(s2) in
// [1/2, 1), D = |alpha| + xn, tau = D / xn, v_i = sgn(alpha) x_i / D.
struct FixRefl {
    ull tau;  // Q62, <= 2^63 - 1
    ull r;    // Q62: 1/D
    ull xn;   // Q62
    int z;
    bool zero;
};

__device__ __forceinline__ FixRefl fix_reflector(unsigned __int128 s2, ll alpha) {
    FixRefl R;
    const ull aa = (ull)(alpha < 0 ? -alpha : alpha);
    R.zero = s2 == (unsigned __int128)aa * aa;
    R.tau = R.r = R.xn = 0;
    R.z = 64;
    if (R.zero) return R;
    const ull top = (ull)(s2 >> 64);
    const int lz = top ? __clzll((ll)top) : 64 + __clzll((ll)(ull)s2);
    const int z = lz & ~1;
    const ull M = (ull)((s2 << z) >> 64);  // Q64, in [1/4, 1)
    constexpr ull kMax = 0x7fffffffffffffffull;
    // y = 1/sqrt(M): Newton (third order) from the FP32 estimate; the estimates go through 32-bit conversions (a
    // 64-bit one takes 64 cycles)
    const float mf = __uint2float_rn((unsigned)(M >> 32)) * 0x1p-32f;
    ull y = min((ull)__float2uint_rn(rsqrtf(mf) * 0x1p30f) << 32, kMax);  // Q62
    {
        const ll e = (1ll << 60) - (ll)__umul64hi(M, __umul64hi(y, y));  // Q60: 1 - M y^2
        const ll e2 = ((e >> 10) * (e >> 10)) >> 40;
        y = min(y + (ull)__mul64hi((ll)y, ((e >> 1) + ((3 * e2) >> 3)) << 4), kMax);
    }
    const ull xn = __umul64hi(M, y);               // Q62: sqrt(M)
    const ull D = (aa << (z / 2 - 2)) + xn;        // Q62, in [1/2, 2)
    const float df = __uint2float_rn((unsigned)(D >> 32)) * 0x1p-30f;
    ull r = min((ull)__float2uint_rn(__fdividef(1.f, df) * 0x1p30f) << 32, kMax);
    {
        const ll e = (1ll << 60) - (ll)__umul64hi(D, r);
        const ll e2 = ((e >> 10) * (e >> 10)) >> 40;
        r = min(r + (ull)__mul64hi((ll)r, (e + e2) << 4), kMax);
    }
    R.tau = min(__umul64hi(D, y) << 2, kMax);
    R.r = r;
    R.xn = xn;
    R.z = z;
    return R;
}

// bytes of the per-CTA arrays ahead of the tiles
struct Smem {
    size_t vp, wp, v, x, pex, pw, nslot, cpart, cslot, pvslot, tab, tiles;
};
template <class P, int NB>
__host__ __device__ inline Smem smem_layout(int max_ld, int C, int max_slots) {
    Smem m;
    size_t o = 0;
    auto take = [&](size_t bytes) {
        const size_t at = o;
        o += (bytes + 15) / 16 * 16;
        return at;
    };
    m.vp = take(sizeof(typename P::V) * max_ld * NB);
    m.wp = take(sizeof(typename P::V) * max_ld * NB);
    m.v = take(sizeof(typename P::V) * max_ld);
    m.x = take(8 * (size_t)max_ld);  // also the build's row sums (doubles)
    m.pex = take(sizeof(typename P::S) * max_ld * C);
    m.pw = take(4 * (size_t)P::kPwWords * max_ld);
    m.nslot = take(3 * 8 * kMaxTileRows);
    m.cpart = take(sizeof(typename P::S) * P::kWarps * 2 * NB);
    m.cslot = take(sizeof(typename P::S) * C * 2 * NB);
    m.pvslot = take(sizeof(typename P::S) * C * P::kWarps);
    m.tab = take(2 * (size_t)max_slots);
    m.tiles = o;
    return m;
}
__host__ __device__ inline int slots_of(int nt, int C) { return (nt * (nt + 1) / 2 + C - 1) / C; }

template <class P, int NB>
__global__ void __launch_bounds__(P::kWarps * 32, P::kOcc)
sytrd_cluster_kernel(const ChainDesc* __restrict__ descs, const double* __restrict__ diag,
                     typename P::G* __restrict__ Aout, void* __restrict__ spill, double* __restrict__ dout,
                     double* __restrict__ eout, typename P::G* __restrict__ tauout, const int* __restrict__ order,
                     int norder, int* __restrict__ counter, int* __restrict__ status, int max_ld, int max_slots,
                     int cap) {
    using V = typename P::V;
    using S = typename P::S;
    using Acc = typename P::Acc;
    constexpr int kWarps = P::kWarps, kThreads = kWarps * 32;
    constexpr bool kFix = sizeof(S) == 8;
    constexpr size_t kTileBytes = sizeof(V) * kTileElems;
    extern __shared__ __align__(16) unsigned char sm[];
    __shared__ int s_item;
    __shared__ double s_red[kWarps], s_rowsum;
    __shared__ FixRefl s_refl;
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int inv_c = 65536 / C + 1;  // exact quotients by C below 8192
    auto div_c = [&](int x) { return x * inv_c >> 16; };
    auto mod_c = [&](int x) { return x - div_c(x) * C; };
    auto first_of = [&](int x) {  // distance from item x to the next one that belongs to this CTA
        const int o = rank - mod_c(x);
        return o < 0 ? o + C : o;
    };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const Smem L = smem_layout<P, NB>(max_ld, C, max_slots);
    V* Vp = (V*)(sm + L.vp);  // [ld][NB]
    V* Wp = (V*)(sm + L.wp);  // [ld][NB]
    V* vv = (V*)(sm + L.v);
    S* xb = (S*)(sm + L.x);
    S* pex = (S*)(sm + L.pex);  // [C][max_ld]
    int* pwi = (int*)(sm + L.pw);
    float* pwf = (float*)(sm + L.pw);
    ll* nslot = (ll*)(sm + L.nslot);   // column norm: [tile row][3] (Fix), [tile row] floats (F32)
    S* cpart = (S*)(sm + L.cpart);     // [warp][2 NB]
    S* cslot = (S*)(sm + L.cslot);     // [CTA][2 NB]
    S* pvslot = (S*)(sm + L.pvslot);   // [CTA][warp]
    unsigned short* tab = (unsigned short*)(sm + L.tab);
    auto csync = [&]() {
        if (C > 1) cl.sync();
        else __syncthreads();
    };
    auto at = [&](auto* p, int r) { return C > 1 ? cl.map_shared_rank(p, r) : p; };

    // the list's items go into every CTA's shared memory: only a CTA that runs has one
    if (order) csync();
    for (int item = blockIdx.x / C;;) {
        if (order) {
            __syncthreads();
            if (rank == 0 && tid == 0) {
                const int it = atomicAdd(counter, 1);
#pragma unroll 1
                for (int r = 0; r < C; ++r) *at(&s_item, r) = it;
            }
            csync();
            item = s_item;
            if (item >= norder) return;
        }
        const ChainDesc D = descs[order ? order[item] : item];
        const int n = D.n, ld = D.ld, nt = ld / kTile;
        typename P::G* __restrict__ A = Aout + D.a_off;
        unsigned char* gt = (unsigned char*)spill + (size_t)D.a_off * sizeof(V);
        const int ntiles = nt * (nt + 1) / 2;
        const int nslots = div_c(ntiles - rank + C - 1);
        auto tile = [&](int slot) -> unsigned char* {
            return slot < cap ? sm + L.tiles + (size_t)slot * kTileBytes : gt + (size_t)(slot * C + rank) * kTileBytes;
        };

        // ---- build: zero the tiles, then scatter H = hopping + diag(-mu_c + U f) ----
#pragma unroll 1
        for (int slot = warp; slot < nslots; slot += kWarps) {
            int4* t = (int4*)tile(slot);
#pragma unroll 1
            for (int q = lane; q < (int)(kTileBytes / 16); q += 32) t[q] = make_int4(0, 0, 0, 0);
            if (lane == 0) {  // tile id -> (I, J): column J holds ids (nt-1-J)(nt-J)/2 ...
                const int id = slot * C + rank;
                int m = (int)((sqrtf(8.f * id + 1.f) - 1.f) * 0.5f);
                while (m * (m + 1) / 2 > id) --m;
                while ((m + 1) * (m + 2) / 2 <= id) ++m;
                const int J = nt - 1 - m, I = J + id - m * (m + 1) / 2;
                tab[slot] = (unsigned short)(I << 8 | J);
            }
        }
#pragma unroll 1
        for (int i = tid; i < ld * NB; i += kThreads) Vp[i] = Wp[i] = P::vzero();
#pragma unroll 1
        for (int i = tid; i < ld; i += kThreads) vv[i] = P::vzero();
#pragma unroll 1
        for (int i = tid; i < P::kPwWords * max_ld; i += kThreads) pwi[i] = 0;
        // Fix: S = 2^eS above the largest absolute row sum of the lower triangle mirrored
        int eS = 0;
        double quant = 1.0, inv = 1.0;
        if constexpr (kFix) {
            double* rs = (double*)xb;
#pragma unroll 1
            for (int i = tid; i < ld; i += kThreads) rs[i] = 0.0;
            __syncthreads();
#pragma unroll 1
            for (int i = tid; i < n; i += kThreads) {
                double own = fabs(diag[D.v_off + i]);
#pragma unroll 1
                for (int q = D.rowptr[i]; q < D.rowptr[i + 1]; ++q) {
                    const int j = D.col[q];
                    if ((unsigned)j > (unsigned)i) continue;
                    const double a = fabs(D.val[q]);
                    own += a;
                    if (j < i) atomicAdd(&rs[j], a);
                }
                atomicAdd(&rs[i], own);
            }
            __syncthreads();
            double m = 0.0;
            bool bad = false;
#pragma unroll 1
            for (int i = tid; i < n; i += kThreads) {
                m = fmax(m, rs[i]);
                bad = bad || !(rs[i] < 0x1p900);
            }
            m = block_max(m, s_red);
            if (__syncthreads_or(bad)) m = NAN;
            // The row sums' rounding depends on the order of the additions, and so, next to a power of two, does the
            // scale: every CTA takes CTA 0's.
            if (rank == 0 && tid == 0)
#pragma unroll 1
                for (int r = 0; r < C; ++r) *at(&s_rowsum, r) = m;
            csync();
            m = s_rowsum;
            if (!(m < 0x1p900)) {  // NaN, Inf or out of the format's range
                if (rank == 0) {
                    if (tid == 0 && status) atomicOr(status, kStatusNaN);
#pragma unroll 1
                    for (int i = tid; i < n; i += kThreads) {
                        dout[D.v_off + i] = NAN;  // and so every eigenvalue and logZ
                        eout[D.v_off + i] = 0.0;
                        tauout[D.v_off + i] = 0;
                    }
                }
                if (!order) return;
                continue;  // every CTA has read its item: CTA 0 writes the next one
            }
            eS = m > 0x1p-900 ? ilogb(m * (1.0 + 0x1p-30)) + 1 : -899;
            quant = scalbn(1.0, eS - 30 - P::kLo);
            inv = scalbn(1.0, 30 + P::kLo - eS);
        }
        __syncthreads();
        auto owner_slot = [&](int I, int J) {  // slot of tile (I, J) if this CTA owns it, else -1
            const int id = (nt - 1 - J) * (nt - J) / 2 + I - J;
            return mod_c(id) == rank ? div_c(id) : -1;
        };
        auto add_elem = [&](int i, int j, double a) {
            const int I = i >> 5, J = j >> 5, slot = owner_slot(I, J);
            if (slot < 0) return;
            unsigned char* t = tile(slot);
#pragma unroll 1
            for (int side = 0; side < (I == J && i != j ? 2 : 1); ++side) {  // diagonal tiles hold both triangles
                const int off = side ? elem_off(j & 31, i & 31) : elem_off(i & 31, j & 31);
                if constexpr (kFix) P::put(t, off, P::split(P::join(P::get(t, off)) + __double2ll_rn(a * inv)));
                else P::put(t, off, P::get(t, off) + (float)a);
            }
        };
#pragma unroll 1
        for (int i = tid; i < n; i += kThreads) {
#pragma unroll 1
            for (int q = D.rowptr[i]; q < D.rowptr[i + 1]; ++q) {
                const int j = D.col[q];
                if ((unsigned)j >= (unsigned)n) {  // a column outside [0, n): skipped, the call fails
                    if (status && rank == 0) atomicOr(status, kStatusBadArg);
                    continue;
                }
                if (j <= i) add_elem(i, j, D.val[q]);
            }
            add_elem(i, i, diag[D.v_off + i]);
        }
        csync();  // no CTA writes into another one that is still building

        // of tile column J: this CTA's first tile row (from J) and its slot; of the live tiles from row I0: their number
        // and the first row. They change every 32 columns.
        int at_J = -1, first_J = 0, slot_J = 0, at_I0 = -1, active = 0, first_I0 = 0;
#pragma unroll 1
        for (int k0 = 0; k0 < n - 2; k0 += NB) {
            const int nbk = min(NB, n - 2 - k0);
#pragma unroll 1
            for (int j = 0; j < nbk; ++j) {
                const int k = k0 + j, s = k + 1, J = k >> 5, kc = k & 31;
                // ---- (1) column k with the panel's pending updates, to every CTA ----
                {
                    if (J != at_J) {
                        const int id0 = (nt - 1 - J) * (nt - J) / 2;
                        at_J = J;
                        first_J = J + first_of(id0);
                        slot_J = div_c(id0 + first_J - J);
                    }
                    int slot = slot_J + warp;
                    V vk[NB], wk[NB];
                    ld_row<NB>(Vp + k * NB, vk);
                    ld_row<NB>(Wp + k * NB, wk);
#pragma unroll 1
                    for (int I = first_J + C * warp; I < nt; I += C * kWarps, slot += kWarps) {
                        const unsigned char* t = tile(slot);
                        const int i = I * kTile + lane;
                        Acc u;
                        P::zero(u);
                        if (j > 0) {
                            V vr[NB], wr[NB];
                            ld_row<NB>(Vp + i * NB, vr);
                            ld_row<NB>(Wp + i * NB, wr);
#pragma unroll
                            for (int l = 0; l < NB; ++l)
                                if (l < j) P::mac2(u, vr[l], wk[l], wr[l], vk[l]);
                        }
                        const V a = P::get(t, elem_off(lane, kc));
                        S x;
                        if constexpr (kFix) x = P::upd_ll(a, u);
                        else x = P::upd(a, u);
                        if (i == k) *(S*)(dout + D.v_off + k) = x;
                        const bool in = i >= s && i < n;
                        if (in)
#pragma unroll 1
                            for (int r = 0; r < C; ++r) *at(&xb[i], r) = x;
                        if constexpr (kFix) {
                            const V xv = in ? P::split(x) : P::vzero();
                            const ll hh = warp_sum_ll((ll)xv.x * xv.x), hl = warp_sum_ll((ll)xv.x * xv.y);
                            const ll l2 = warp_sum_ll((ll)xv.y * xv.y);
                            if (lane < C) {
                                ll* d = at(&nslot[3 * (I - J)], lane);
                                d[0] = hh; d[1] = hl; d[2] = l2;
                            }
                        } else {
                            const float q = warp_sum(in && i > s ? x * x : 0.f);
                            if (lane < C) *at((float*)nslot + (I - J), lane) = q;
                        }
                    }
                }
                csync();
                // ---- (2) reflector (every warp forms the same scalars) ----
                const int nact = nt - J;
                bool flat;
                float tau = 0.f, beta = 0.f, scale = 0.f;
                FixRefl R;
                const S alpha = xb[s];
                if constexpr (kFix) {
                    // one warp forms the scalars (~300 instructions), the others wait
                    if (warp == 0) {
                        ll hh = 0, hl = 0, l2 = 0;
                        if (lane < nact) { hh = nslot[3 * lane]; hl = nslot[3 * lane + 1]; l2 = nslot[3 * lane + 2]; }
                        hh = warp_sum_ll(hh);
                        hl = warp_sum_ll(hl);
                        l2 = warp_sum_ll(l2);
                        const unsigned __int128 s2 = ((unsigned __int128)(ull)hh << (2 * P::kLo)) +
                                                     (unsigned __int128)((__int128)hl << (P::kLo + 1)) + (ull)l2;
                        R = fix_reflector(s2, alpha);
                        if (lane == 0) s_refl = R;
                    }
                    __syncthreads();
                    R = s_refl;
                    flat = R.zero;
                } else {
                    const float sigma = warp_sum(lane < nact ? ((const float*)nslot)[lane] : 0.f);
                    beta = alpha;
                    flat = sigma == 0.f;
                    if (!flat) {
                        const float xnorm = sqrtf(alpha * alpha + sigma);
                        beta = alpha >= 0.f ? -xnorm : xnorm;
                        tau = (beta - alpha) / beta;
                        scale = 1.f / (alpha - beta);
                    }
                }
                if (rank == 0 && tid == 0) {  // raw; converted after the last column (FP64 pipe)
                    if constexpr (kFix) {
                        // 2^-62 S: sqrt(s2) has at most 62 bits there
                        const int sh = R.z / 2 - 34 + P::kLo;
                        const ll xn = (ll)(sh >= 0 ? R.xn >> sh : R.xn << -sh);
                        *(ll*)(eout + D.v_off + k) = flat ? alpha << (32 - P::kLo) : (alpha >= 0 ? -xn : xn);
                        if (Aout) *(ull*)(tauout + D.v_off + k) = R.tau;
                    } else {
                        *(float*)(eout + D.v_off + k) = beta;
                        tauout[D.v_off + k] = tau;
                    }
                }
#pragma unroll 1
                for (int i = (k0 & ~31) + tid; i < ld; i += kThreads) {
                    V vi = P::vzero();
                    if (!flat && i >= s && i < n) {
                        if constexpr (kFix) {
                            ll v = 1ll << (30 + P::kLo);
                            if (i > s) {
                                v = P::template round_to<61, 30 + P::kLo>(__mul64hi(xb[i] << (R.z / 2 - 1), (ll)R.r));
                                if (alpha < 0) v = -v;
                            }
                            vi = P::split(v);
                        } else {
                            vi = i == s ? 1.f : xb[i] * scale;
                        }
                    }
                    vv[i] = vi;
                    Vp[i * NB + j] = vi;
                    if (flat) Wp[i * NB + j] = P::vzero();
                    if ((!kFix || Aout) && i > s && i < n && mod_c(i >> 5) == rank) {
                        if constexpr (kFix) {
                            A[(size_t)k * ld + i] = (double)P::join(vi) * (1.0 / (1ll << (30 + P::kLo)));
                        } else {
                            A[(size_t)k * ld + i] = vi;
                        }
                    }
                }
                if (flat) {
                    csync();  // xb and nslot are rewritten by the next column
                    continue;
                }
                __syncthreads();
                // ---- (3a) partial p = A22 v over this CTA's tiles (stale trailing matrix) ----
                const int I0 = s >> 5;
                if (I0 != at_I0) {
                    const int ntr = nt - I0;
                    at_I0 = I0;
                    active = div_c(ntr * (ntr + 1) / 2 - rank + C - 1);
                    first_I0 = I0 + first_of(I0);
                }
                {
                    const int per = (active + kWarps - 1) / kWarps;
                    const int b0 = warp * per, b1 = min(active, b0 + per);
                    auto flush = [&](int i, S p) {
                        if constexpr (kFix) {
                            atomicAdd(&pwi[3 * i], (int)(p & 0x1fffff));
                            atomicAdd(&pwi[3 * i + 1], (int)((p >> 21) & 0x1fffff));
                            atomicAdd(&pwi[3 * i + 2], (int)(p >> 42));
                        } else {
                            __syncwarp();  // another lane may have added to this entry in the flush before
                            pwf[warp * max_ld + i] += p;
                        }
                    };
                    Acc cs[8];
                    V vc[8];
                    int Jc = -1;
#pragma unroll 1
                    for (int unit = b0; unit <= b1; ++unit) {
                        const int ij = unit < b1 ? tab[unit] : 255, I = ij >> 8, Jt = ij & 255;
                        if (Jt != Jc) {
                            if (Jc >= 0) {  // the column sums of the finished tile column
                                S x[8];
#pragma unroll
                                for (int m = 0; m < 8; ++m) x[m] = P::sum(cs[m]);
                                int idx;
                                const S p = reduce_scatter<8, 16>(x, lane, idx);
                                flush(Jc * kTile + (idx >> 1) * 8 + 2 * t4 + (idx & 1), p);
                            }
                            if (unit == b1) break;
                            Jc = Jt;
#pragma unroll
                            for (int m = 0; m < 8; ++m) P::zero(cs[m]);
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                V w2[2];
                                P::ld2(vv + Jt * kTile + q * 8 + 2 * t4, w2);
                                vc[2 * q] = w2[0];
                                vc[2 * q + 1] = w2[1];
                            }
                        }
                        const void* t = tile(unit);
                        S x[4];
#pragma unroll
                        for (int mt = 0; mt < 2; ++mt) {
                            V vr[2];
                            Acc rs[2];
#pragma unroll
                            for (int h = 0; h < 2; ++h) {  // a diagonal tile holds both triangles: row sums only
                                vr[h] = I == Jt ? P::vzero() : vv[I * kTile + 16 * mt + 8 * h + g];
                                P::zero(rs[h]);
                            }
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                V a[4];
                                P::ld4(t, 4 * mt + q, lane, a);
#pragma unroll
                                for (int h = 0; h < 2; ++h) {
                                    P::mac2(rs[h], a[2 * h], vc[2 * q], a[2 * h + 1], vc[2 * q + 1]);
                                    P::mac2(cs[2 * q + h], a[h], vr[0], a[2 + h], vr[1]);
                                }
                            }
                            x[2 * mt] = P::sum(rs[0]);
                            x[2 * mt + 1] = P::sum(rs[1]);
                        }
                        int idx;
                        const S p = reduce_scatter<4, 2>(x, lane, idx);
                        flush(I * kTile + 8 * idx + g, p);
                    }
                }
                // ---- (3b) c1 = W^T v, c2 = V^T v over this CTA's tile rows ----
                if (j > 0) {
                    Acc cacc[2 * NB];
#pragma unroll
                    for (int l = 0; l < 2 * NB; ++l) P::zero(cacc[l]);
#pragma unroll 1
                    for (int I = first_I0 + C * (kWarps - 1 - warp); I < nt; I += C * kWarps) {
                        const int i = I * kTile + lane;
                        const V vi = vv[i];
                        V vr[NB], wr[NB];
                        ld_row<NB>(Vp + i * NB, vr);
                        ld_row<NB>(Wp + i * NB, wr);
#pragma unroll
                        for (int l = 0; l < NB; ++l)
                            if (l < j) {
                                P::mac(cacc[l], wr[l], vi);
                                P::mac(cacc[NB + l], vr[l], vi);
                            }
                    }
                    S x[2 * NB];
#pragma unroll
                    for (int l = 0; l < 2 * NB; ++l) x[l] = P::sum(cacc[l]);
                    int idx;
                    S tot = reduce_scatter<2 * NB, 16>(x, lane, idx);
#pragma unroll
                    for (int o2 = 16 / (2 * NB); o2 >= 1; o2 >>= 1)
                        tot = add_mod(tot, __shfl_xor_sync(0xffffffffu, tot, o2));
                    if ((lane & (32 / (2 * NB) - 1)) == 0) cpart[warp * 2 * NB + idx] = tot;
                }
                __syncthreads();
                // ---- (3c) the partial sums to every CTA ----
                {
                    Acc pv;
                    P::zero(pv);
#pragma unroll 1
                    for (int i = I0 * kTile + tid; i < ld; i += kThreads) {
                        S p;
                        if constexpr (kFix) {
                            const int a0 = pwi[3 * i], a1 = pwi[3 * i + 1], a2 = pwi[3 * i + 2];
                            pwi[3 * i] = pwi[3 * i + 1] = pwi[3 * i + 2] = 0;
                            p = (ll)((ull)(ll)a0 + ((ull)(ll)a1 << 21) + ((ull)(ll)a2 << 42));  // units 2^-60 S
                            P::mac(pv, P::split(P::template round_to<60, 30 + P::kLo>(p)), vv[i]);
                        } else {
                            p = 0.f;
#pragma unroll
                            for (int w = 0; w < kWarps; ++w) {
                                p += pwf[w * max_ld + i];
                                pwf[w * max_ld + i] = 0.f;
                            }
                            P::mac(pv, p, vv[i]);
                        }
#pragma unroll 1
                        for (int r = 0; r < C; ++r) at(pex, r)[rank * max_ld + i] = p;
                    }
                    S pvs = P::sum(pv);
                    if constexpr (kFix) pvs = warp_sum_ll(pvs);
                    else pvs = warp_sum(pvs);
                    if (lane < C) at(pvslot, lane)[rank * kWarps + warp] = pvs;
                    if (j > 0 && tid < 2 * NB) {
                        S c = 0;
#pragma unroll 1
                        for (int w = 0; w < kWarps; ++w) c = add_mod(c, cpart[w * 2 * NB + tid]);
#pragma unroll 1
                        for (int r = 0; r < C; ++r) at(cslot, r)[rank * 2 * NB + tid] = c;
                    }
                }
                csync();
                // ---- (4) w = tau p - (tau/2)(tau p . v) v with p corrected by V and W ----
                {
                    V c1[NB], c2[NB];
#pragma unroll
                    for (int l = 0; l < NB; ++l) c1[l] = c2[l] = P::vzero();
                    S pv = 0;
#pragma unroll 1
                    for (int q = lane; q < C * kWarps; q += 32) pv = add_mod(pv, pvslot[q]);
                    if constexpr (kFix) pv = warp_sum_ll(pv);
                    else pv = warp_sum(pv);
                    if (j > 0) {
                        S c = 0;
                        if (lane < 2 * NB)
#pragma unroll 1
                            for (int r = 0; r < C; ++r) c = add_mod(c, cslot[r * 2 * NB + lane]);
                        Acc cc;
                        P::zero(cc);
#pragma unroll
                        for (int l = 0; l < NB; ++l) {
                            const S a = __shfl_sync(0xffffffffu, c, l), b = __shfl_sync(0xffffffffu, c, NB + l);
                            if constexpr (kFix) {
                                c1[l] = P::split(P::template round_to<59, 28 + P::kLo>(a));
                                c2[l] = P::split(P::template round_to<60, 29 + P::kLo>(b));
                            } else {
                                c1[l] = a;
                                c2[l] = b;
                            }
                            if (l >= j) c1[l] = c2[l] = P::vzero();
                            P::mac(cc, c1[l], c2[l]);
                        }
                        // p . v = v^T A v - 2 c1 . c2 (c1 c2 in units 2^-57 S)
                        if constexpr (kFix) pv -= P::sum(cc) << 4;
                        else pv -= 2.f * cc.s;
                    }
                    float K = 0.f;
                    V Kv;
                    if constexpr (kFix) {
                        Kv = P::k_value(pv, (ll)R.tau);
                    } else {
                        K = 0.5f * tau * (tau * pv);
                        Kv = K;
                    }
#pragma unroll 1
                    for (int i = (k0 & ~31) + tid; i < ld; i += kThreads) {
                        V w = P::vzero();
                        if (i >= s && i < n) {
                            S q = pex[i];
#pragma unroll 1
                            for (int r = 1; r < C; ++r) q = add_mod(q, pex[r * max_ld + i]);
                            Acc u;
                            P::zero(u);
                            if (j > 0) {
                                V vr[NB], wr[NB];
                                ld_row<NB>(Vp + i * NB, vr);
                                ld_row<NB>(Wp + i * NB, wr);
#pragma unroll
                                for (int l = 0; l < NB; ++l)
                                    if (l < j) P::mac2(u, vr[l], c1[l], wr[l], c2[l]);
                            }
                            if constexpr (kFix) {
                                q -= P::sum(u) << 2;  // 2^-58 S -> 2^-60 S
                                Acc kv;
                                P::zero(kv);
                                P::mac(kv, Kv, vv[i]);  // 2^-59 S
                                w = P::w_entry(q, (ll)R.tau, kv);
                            } else {
                                w = tau * (q - u.s) - K * vv[i];
                            }
                        }
                        Wp[i * NB + j] = w;
                    }
                }
                __syncthreads();
            }
            // ---- (5) A22 -= V W^T + W V^T over this CTA's live tiles ----
            if (nbk < NB) {
#pragma unroll 1
                for (int i = tid; i < ld; i += kThreads)
                    for (int l = nbk; l < NB; ++l) Vp[i * NB + l] = Wp[i * NB + l] = P::vzero();
                __syncthreads();
            }
            {
                const int I0 = (k0 + nbk) >> 5, ntr = nt - I0, total = ntr * (ntr + 1) / 2;
                const int active = div_c(total - rank + C - 1);
#pragma unroll 1
                for (int unit = warp; unit < 2 * active; unit += kWarps) {  // 16 rows of a tile
                    const int ij = tab[unit >> 1], I = ij >> 8, Jt = ij & 255, mt = unit & 1;
                    void* t = tile(unit >> 1);
                    V a[4][4], vr[2][NB], wr[2][NB];
#pragma unroll
                    for (int q = 0; q < 4; ++q) P::ld4(t, mt * 4 + q, lane, a[q]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        ld_row<NB>(Vp + (I * kTile + 16 * mt + 8 * h + g) * NB, vr[h]);
                        ld_row<NB>(Wp + (I * kTile + 16 * mt + 8 * h + g) * NB, wr[h]);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
#pragma unroll
                        for (int c = 0; c < 2; ++c) {
                            V cv[NB], cw[NB];
                            ld_row<NB>(Vp + (Jt * kTile + 8 * q + 2 * t4 + c) * NB, cv);
                            ld_row<NB>(Wp + (Jt * kTile + 8 * q + 2 * t4 + c) * NB, cw);
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                Acc u;
                                P::zero(u);
#pragma unroll
                                for (int l = 0; l < NB; ++l) P::mac2(u, vr[h][l], cw[l], wr[h][l], cv[l]);
                                a[q][2 * h + c] = P::upd(a[q][2 * h + c], u);
                            }
                        }
                        P::st4(t, mt * 4 + q, lane, a[q]);
                    }
                }
            }
            __syncthreads();
        }
        // ---- the trailing 2 x 2 block (n <= 2: the whole matrix), then the outputs ----
        if (tid == 0) {
#pragma unroll 1
            for (int e = 0; e < 3; ++e) {
                const int i = n - 2 + (e >> 1), jj = e == 1 ? i + 1 : i;  // (n-2, n-2), (n-1, n-2), (n-1, n-1)
                const int slot = i < 0 ? -1 : owner_slot(jj >> 5, i >> 5);
                if (slot < 0) continue;
                const V a = P::get(tile(slot), elem_off(jj & 31, i & 31));
                S* o = (S*)((e == 1 ? eout : dout) + D.v_off + i);
                if constexpr (kFix) *o = P::join(a) << (e == 1 ? 32 - P::kLo : 0);
                else *o = a;
            }
        }
        csync();
        if (rank == 0)
#pragma unroll 1
            for (int i = tid; i < n; i += kThreads) {
                double* d = dout + D.v_off + i;
                double* e = eout + D.v_off + i;
                if constexpr (kFix) {
                    *d = (double)__ldcg((ll*)d) * quant;
                    if (i < n - 1) *e = (double)__ldcg((ll*)e) * (quant / (1ll << (32 - P::kLo)));
                    double* t = tauout + D.v_off + i;
                    if (Aout && i < n - 2) *t = (double)__ldcg((ull*)t) * 0x1p-62;
                } else {
                    *d = (double)__ldcg((float*)d);
                    if (i < n - 1) *e = (double)__ldcg((float*)e);
                }
                if (i == n - 2) tauout[D.v_off + i] = 0;
            }
        if (!order) return;
    }
}

}  // namespace

// Cluster size (any of 1 .. 8) and grid of a launch. The time of one chain's column was fitted on the GPU (one chain
// per cluster) as P::kCost has it: FP64 over N = 64 .. 1024; FP32 for each number of warps over N = 130 .. 1024 and C = 1
// .. 8, 2 % rms, and two CTAs on an SM 14 .. 24 % slower than one (one set for all warps took C = 8 where 1 or 4 is better: 32 chains of N = 216 0.86 -> 0.70 ms, one of
// N = 256 0.94 -> 0.88). `fit` clusters run at once (152, 76, 36, 15 for C = 1, 2, 4, 8). Measured ms behind the choice (C =
// 1, 2, 4, 8), FP64 path: 256 chains of N = 576 30.4, 34.2, 46.6, 85; 16 chains 13.8, 8.6, 5.9, 9.5 (two rounds); one
// chain of N = 343 4.2, 3.0, 2.4, 2.1. FP32: 256 chains of N = 576 7.9, 12.8, 21.3, 47.6; 16 chains of N = 1024 15.3, 10.1,
// 7.4, 12.7.
template <class P>
static double cluster_cost(int n, int nt, int C, int cap) {
    constexpr ColumnCost k = P::kCost;
    const double share = nt * (nt + 1) / 2 / (3.0 * C), spilled = max(0, slots_of(nt, C) - cap) / 3.0;
    return n * (k.base + k.row * n + k.tile * share + k.spill * spilled + (C > 1 ? k.cluster + k.cta * (C - 1) : 0.0));
}

template <class P, int NB>
static cudaError_t launch_cluster(const ChainDesc* h_desc, const ChainDesc* d_desc, int batch, int max_ld,
                                  const double* d_diag, typename P::G* d_A, void* d_spill, double* d_d, double* d_e,
                                  typename P::G* d_tau, const int* d_order, int* d_counter, int num_sms,
                                  int* d_status, cudaStream_t st) {
    if (batch <= 0) return cudaSuccess;
    auto* kern = sytrd_cluster_kernel<P, NB>;
    const size_t tile_bytes = sizeof(typename P::V) * kTileElems, limit = 226 * 1024 / P::kOcc;
    // the attribute belongs to the process: one value, whatever another thread's context launches meanwhile
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
    if (err != cudaSuccess) return err;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.blockDim = dim3(P::kWarps * 32);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int best_slots = 0, best_cap = 0, best_fit = 0, best_C = 0;
    size_t best_smem = 0;
    double best = 0.0;
    // from the largest down: with the fewest chains the first is the best, and the others need no query
    for (int C = d_order ? 8 : 1; C >= 1; --C) {
        const int slots = slots_of(max_ld / kTile, C);
        const size_t head = smem_layout<P, NB>(max_ld, C, slots).tiles;
        if (head > limit) continue;
        const int cap = (int)min((size_t)slots, (limit - head) / tile_bytes);
        if (cap < slots && !d_spill) continue;
        const size_t smem = head + cap * tile_bytes;
        int fit = batch;
        double cost = 0.0;
        if (d_order) {
            double sum = 0.0, mx = 0.0, mn = 1e300;
            for (int c = 0; c < batch; ++c) {
                const double t = cluster_cost<P>(h_desc[c].n, h_desc[c].ld / kTile, C, cap);
                sum += t;
                mx = max(mx, t);
                mn = min(mn, t);
            }
            // equal chains run in whole rounds, uneven ones (longest first) end within about half the longest
            auto total = [&](int f) {
                const int ctas = (min(batch, f) * P::kOcc + f - 1) / f;  // on the fullest SM
                return (mn == mx ? mx * ((batch + f - 1) / f) : max(mx, sum / f + 0.5 * mx)) *
                       (1.0 + P::kCost.shared * (ctas - 1));
            };
            if (best_C && total(max(1, num_sms * P::kOcc / C)) >= best) continue;
            at.val.clusterDim.x = C;
            cfg.gridDim = dim3(batch * C);
            cfg.dynamicSmemBytes = smem;
            if ((err = cudaOccupancyMaxActiveClusters(&fit, kern, &cfg))) return err;
            if (fit < 1) continue;
            cost = total(fit);
        }
        if (best_C && cost >= best) continue;
        best = cost;
        best_C = C;
        best_slots = slots;
        best_cap = cap;
        best_fit = fit;
        best_smem = smem;
    }
    if (!best_C) return cudaErrorInvalidValue;
    if (d_order && (err = cudaMemsetAsync(d_counter, 0, sizeof(int), st))) return err;
    at.val.clusterDim.x = best_C;
    cfg.gridDim = dim3(min(batch, best_fit) * best_C);
    cfg.dynamicSmemBytes = best_smem;
    return cudaLaunchKernelEx(&cfg, kern, d_desc, d_diag, d_A, d_spill, d_d, d_e, d_tau, d_order, batch, d_counter,
                              d_status, max_ld, best_slots, best_cap);
}

}  // namespace fkg
