// fd1d_onchip.cuh -- the on-chip theta-scheme kernel: one, two or four warps per PDE, the
// whole PDE in registers and shared memory, stepping in FP32.  Two modes:
//   kPair = false (fd1d_fp32.cu): one FP32 solve per step for the increment, V less the payoff
//     as an unevaluated pair of floats;
//   kPair = true (fd1d_pair64.cu): two solves per step and a residual in pair arithmetic --
//     FP64 accuracy, theta = 1/2.
//
// Solve of B u = r: lane K owns nodes K M .. K M + M - 1, node K M is a separator, the others
// are eliminated from both ends towards the lane's pivot node P = M / 2 (two chains of M/2 - 1
// steps), spikes couple them to the separators, and the separator system is solved by
// cyclic reduction over the warp.  With W > 1 warps per PDE each warp reduces its own 32
// separators, and the 2 (W - 1) values at the warp boundaries come from one dense product
// with the inverse of their system (one block barrier per solve instead of one per
// reduction level).
//
// Packed pairs.  Every step runs on float2 values with the packed FP32 instructions of sm_100
// and later: nodes P-k and P+k share a float2 (slot k; slot 0 holds nodes 0 and P).  Measured
// on the card, a packed operation holds the FP32 pipe as long as two scalar ones (2.13 cycles
// per warp and scheduler) and takes one issue slot instead of two; negating an operand is
// free.  The per-node work is the same for any pairing; this one also packs the two
// elimination chains.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "fd1d_common.cuh"
#include "fd1d_kernels.h"

namespace kwg {

namespace {

constexpr unsigned kAll = 0xffffffffu;
// Separators whose multipliers are below this (2^-45) no longer see each other.
constexpr float kNoCoupling = 2.8e-14f;
// Payoffs and coefficients above this leave no room for the pair arithmetic in FP32's range.
constexpr double kMaxValue = 1e30;

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg(b)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// s + e = a + b exactly, and s + e = a - b exactly (Knuth), for any magnitudes.
__device__ __forceinline__ void two_sum(float2 a, float2 b, float2& s, float2& e)
{
    s = add2(a, b);
    const float2 bb = sub2(s, a);
    e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}
__device__ __forceinline__ void two_diff(float2 a, float2 b, float2& s, float2& e)
{
    s = sub2(a, b);
    const float2 bb = sub2(s, a);
    e = sub2(sub2(a, sub2(s, bb)), add2(b, bb));
}

// Keeps the compiler from loading the next phase's tables ahead of time: with one warp per
// PDE no barrier stands between the phases, and the loads it moved up cost registers (pair
// arithmetic, M = 32: 255 and 444 bytes of spills without, 218 and none with).  Where registers
// are to spare the early loads are worth 3 to 10 %.
template <bool kOn>
__device__ __forceinline__ void phase_edge()
{
    if constexpr (kOn) __syncwarp();
}

// A pair of values, each an unevaluated sum hi + lo.
struct PP2 {
    float2 h, l;
};

// W = V + u as a pair; V.h + u = W.h + e exactly.
__device__ __forceinline__ PP2 shifted(float2 H, float2 L, float2 u)
{
    PP2 w;
    float2 e;
    two_sum(H, u, w.h, e);
    w.l = add2(L, e);
    return w;
}

// a - b of two pairs.
__device__ __forceinline__ PP2 pair_diff(const PP2& a, const PP2& b)
{
    PP2 d;
    float2 e;
    two_diff(a.h, b.h, d.h, e);
    d.l = add2(e, sub2(a.l, b.l));
    return d;
}

// The same with the low part within an ulp of the high one (Fast2Sum; where the difference is below
// 2^-24 of the values the loss is that of pair_diff).  The low parts of neighbouring values do not
// cancel as the values do: as they come, a difference's is up to 2^-24 of the values, and a step's
// residual rounds it times alpha.  2 % of a call; errors against 64-bit stepping before -> after, FD1D-BS at density
// 0.25: 1024 x 1024 1.9e-13 -> 1.0e-14, 1024 x 40 8.4e-13 -> 1.2e-14, 512 x 40 3.4e-13 -> 1.1e-14.
__device__ __forceinline__ PP2 pair_diff_norm(const PP2& a, const PP2& b)
{
    const PP2 d = pair_diff(a, b);
    const float2 h = add2(d.h, d.l);
    return {h, sub2(d.l, sub2(h, d.h))};
}

// alpha X - beta Y + gamma W - u of pairs; the parts cancel, the result is one float.  The
// low parts of X and Y times alpha and beta are the largest of the small terms: they come
// last, so that the rounding of the others stays below theirs (adding them first and
// collecting the rest afterwards gave six times the error on 2048-node sinh grids).
__device__ __forceinline__ float2 pair_residual(float2 ah, float2 al, const PP2& x, float2 bh, float2 bl, const PP2& y,
                                                float2 gh, float2 gl, const PP2& w, float2 u)
{
    const float2 p1 = mul2(ah, x.h), p2 = mul2(bh, y.h), p3 = mul2(gh, w.h);
    const float2 e1 = fma2(al, x.h, fma2(ah, x.h, neg(p1)));
    const float2 e2 = fma2(neg(bl), y.h, fma2(neg(bh), y.h, p2));
    const float2 e3 = fma2(gh, w.l, fma2(gl, w.h, fma2(gh, w.h, neg(p3))));
    float2 s1, t1, s2, t2;
    two_diff(p1, p2, s1, t1);
    two_diff(p3, u, s2, t2);
    const float2 small = add2(add2(e1, e2), add2(e3, add2(t1, t2)));
    return add2(fma2(ah, x.l, add2(s1, s2)), fma2(neg(bh), y.l, small));
}

// (h, l) += d for FP32 stepping: h takes the rounded sum and l collects its rounding error by
// Fast2Sum (exact when |h| >= |d| or h == 0 -- the increment of a step is small next to the
// value it updates; where it is not, X is near 0 and the loss is an ulp of that tiny sum).
// The pair is not renormalised: each step adds at most half an ulp of h to l, so over a
// few thousand steps |l| stays within ~2^11 ulp(h), far below h, and the differences of
// neighbouring h that the residual takes stay exact.
__device__ __forceinline__ void ff_acc2(float2& h, float2& l, float2 d)
{
    const float2 s = add2(h, d);
    l = add2(l, sub2(d, sub2(s, h)));
    h = s;
}

// (h, l) += 2 u + 2 e for pairs, renormalised.
__device__ __forceinline__ void pair_acc2(float2& h, float2& l, float2 u, float2 e)
{
    float2 s, r;
    two_sum(h, add2(u, u), s, r);
    const float2 t = fma2(f2(2.f, 2.f), e, add2(l, r));
    h = add2(s, t);
    l = sub2(t, sub2(h, s));
}

// (h, l) = max((h, l), (ph, pl))
__device__ __forceinline__ void floor_to(float2 ph, float2 pl, float2& h, float2& l)
{
    const float2 d = add2(sub2(h, ph), sub2(l, pl));
    if (d.x < 0.f) {
        h.x = ph.x;
        l.x = pl.x;
    }
    if (d.y < 0.f) {
        h.y = ph.y;
        l.y = pl.y;
    }
}

// 1 / d by one step of Chebyshev's third-order iteration (Newton's with the next term of the series),
// r (1 + e + e^2) with e = 1 - d r, from the hardware's 20-bit estimate: e^3 ~ 2^-60 is left, then
// rounding: within an ulp for d from 2^-1000 to 2^1000.  Zero and non-finite d give a non-finite result.
__device__ __forceinline__ double rcp(double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d, r, 1.);
    return fma(r, fma(e, e, e), r);
}

struct Split {
    float h, l;
};
__device__ __forceinline__ Split split(double v)
{
    Split r;
    r.h = __double2float_rn(v);
    r.l = __double2float_rn(__dsub_rn(v, (double)r.h));
    return r;
}

// A variant's share of the registers: the warps per SM that must fit, phase edges, and how
// many of the factor tables stay in registers for the whole PDE (the spikes; also 1/d and u;
// also l -- shared memory otherwise returns them every step, 40 of 56 bytes per slot and lane in
// FP32 stepping, where it was the busiest unit, 71 %).  Best of 1 to 40 settings each; the tables in registers
// took 2 to 30 % off.  Kernel ms now (511 steps; pair arithmetic at 1024 and 2048 nodes 255), FP32 | pair:
//   M = 32 uniform   8192 x 1024   3.77 | 5.85       M = 8 uniform  16384 x 256   1.94 | 5.85
//   M = 16 uniform   8192 x 512    1.95 | 5.78       M = 8          16384 x 256   2.29 | 6.41
//   M = 16           8192 x 512    2.38 | 6.59       M = 4 uniform  16384 x 128   1.12 | 3.54
//   M = 16, W = 2    8192 x 1024   5.25 | 7.06       M = 4          16384 x 128   1.32 | 3.78
//   M = 16, W = 4    4096 x 2048   5.87 | 7.94       M = 2 uniform  16384 x 64    0.75 | 2.22
// Variants that only small batches take (more warps per PDE than a large batch would) need
// registers, not resident warps: 150 PDEs of 1024 uniform nodes (256 steps) 0.318 -> 0.267 pair; 300 of 2048
// uniform nodes 0.267 -> 0.239 FP32.
struct Budget {
    int warps, tables;
    bool edges;
};
__host__ __device__ constexpr Budget budget(int M, int W, bool uni, bool pair)
{
    if (!pair) {
        if (M == 32) return uni ? Budget{12, 0, W == 1} : Budget{8, 1, W == 2};
        if (M == 16 && uni) return W == 1 ? Budget{12, 2, true} : W == 2 ? Budget{12, 1, false} : Budget{10, 3, false};
        if (M == 16) return W == 4 ? Budget{12, 2, false} : Budget{10, 2, true};
        if (W > 1) return M == 8 && uni && W == 4 ? Budget{10, 3, false} : Budget{12, 3, M == 8};
        if (M == 2) return {20, 0, false};
        return {M == 8 && !uni ? 16 : 20, uni ? 2 : 3, false};
    }
    if (M == 32) return {12, 0, true};
    if (M == 16 && uni) return W == 1 ? Budget{10, 2, true} : W == 2 ? Budget{10, 1, false} : Budget{16, 0, false};
    if (M == 16) return W == 1 ? Budget{8, 3, false} : W == 2 ? Budget{10, 1, false} : Budget{12, 1, false};
    if (M == 8) return {W > 1 ? 12 : 16, 3, true};
    if (M == 4) return W > 1 ? Budget{10, 3, false} : uni ? Budget{16, 3, false} : Budget{20, 3, true};
    return uni ? Budget{16, 3, true} : Budget{10, 3, false};
}

// Shared-memory layout of one PDE group (floats).  P = M / 2 slots, NL = 32 W lanes.
//   PPt  [P][NL] float4   payoff (hi_a, hi_b, lo_a, lo_b), hi -inf where no floor applies; in
//                         FP32 stepping q [P][NL] float2 in its place
//   Cht  [S][NL] float4   (A_a, A_b, B_a, B_b) high parts, Clt low parts: the multipliers
//                         of a slot's two differences (below); S = P, or on uniform grids
//                         of full lanes the two slots that can hold a boundary node
//   T1 (l), T2 (1/d, u), T3 (spikes L, R): the factors, [P][stride]; on uniform grids of
//                         full lanes once for the group and once for the last lane
// then the exchange area of W > 1.
template <int M, bool kUni, int W, bool kPair>
struct Lay {
    static constexpr int P = M / 2, NL = 32 * W;
    static constexpr int S = kUni ? (P > 1 ? 2 : 1) : P;
    static constexpr int kStride = kUni ? 2 : NL;
    static constexpr int oPP = 0;
    static constexpr int oCh = oPP + 4 * P * NL;
    static constexpr int oCl = oCh + 4 * S * NL;
    static constexpr int oT2 = oCl + (kPair ? 4 : 2) * S * NL;
    static constexpr int oT3 = oT2 + 4 * P * kStride;
    static constexpr bool kSpikeRegs = !kUni && budget(M, W, kUni, kPair).tables >= 1;  // no T3
    static constexpr int oT1 = oT3 + (kSpikeRegs ? 0 : 4 * P * kStride);
    static constexpr int oX = oT1 + 2 * P * kStride;
    static constexpr int n = 2 * (W - 1), nv = 3 * (W - 1);  // boundary unknowns and their inputs
    // exchange area: edges [W][4], inputs of the two solves [2][nv], inverse [nv][n],
    // spikes at the warp boundaries [W][2], PDE number and status
    static constexpr int oEdge = oX, oVec = oEdge + 4 * W, oInv = oVec + 2 * (nv + 1), oSp = oInv + nv * n,
                         oInt = oSp + 2 * W;
    static constexpr int kEx = W == 1 ? 0 : 4 * W + 2 * (nv + 1) + nv * n + 2 * W + W + 2;
    // setup exchange in doubles (the payoff table's space is in use): [2][W] spike ends of each warp's
    // last node, [5][W] responses at the warp boundaries
    static constexpr int oDbl = (oX + kEx + 1) / 2 * 2;
    static constexpr int kDbl = W == 1 ? 0 : 2 * 7 * W;
    static constexpr size_t kBytes = (size_t)(oDbl + kDbl) * sizeof(float);
};

}  // namespace

template <int M, bool kUni, int W, bool kPair>
__global__ void __launch_bounds__(32 * W, budget(M, W, kUni, kPair).warps / W)
    fd1d_solve_onchip(const PdeBatch b, Fd1dShape sh, double* __restrict__ vout, int32_t* __restrict__ pde_status,
                      int* __restrict__ counters, int32_t* __restrict__ rescue)
{
    using Y = Lay<M, kUni, W, kPair>;
    constexpr bool kEdge = budget(M, W, kUni, kPair).edges;
    constexpr int kReg = budget(M, W, kUni, kPair).tables;
    // Stop the cyclic reduction at the level where the separators no longer see each other: the multipliers
    // square from level to level, and at 1024 uniform nodes only the first counts.  The branch
    // splits the solve for the compiler's scheduling, so only where it pays: FP32, 16384 PDEs of 64 uniform
    // nodes 0.845 -> 0.745 ms, 128 1.24 -> 1.12, 256 2.00 -> 1.94, 8192 of 1024 3.86 -> 3.78; pair, 16384 of 128
    // 1.83 -> 1.75, 3 of 51 nodes 0.604 -> 0.454.  Not with several warps (128 PDEs of 512 nodes, FP32, 0.200 ->
    // 0.221) or on most grids with tables per node (16384 of 128, 1.32 -> 1.35).
    constexpr bool kCut = W == 1 && (kUni ? !kPair || M < 32 : M == 2 || (M == 16 && !kPair));
    constexpr bool kOwn = W > 1 && (!kPair || M <= 8);  // every lane steps its two neighbour nodes itself
    constexpr int P = Y::P, NL = Y::NL, kStride = Y::kStride;
    static_assert(M >= 2 && M % 2 == 0, "as many rows above the pivot as below");
    extern __shared__ __align__(16) float tab[];
    const int k = threadIdx.x & 31, warp = W == 1 ? 0 : threadIdx.x >> 5;
    const int K = threadIdx.x;
    const int own = kUni ? (K + 1) / NL : K;
    float4* const PPt = reinterpret_cast<float4*>(tab + Y::oPP) + K;
    float4* const Cht = reinterpret_cast<float4*>(tab + Y::oCh) + K;
    float4* const Clt = reinterpret_cast<float4*>(tab + Y::oCl) + K;    // pairs
    float2* const C1t = reinterpret_cast<float2*>(tab + Y::oCl) + K;    // FP32 stepping
    float4* const T2 = reinterpret_cast<float4*>(tab + Y::oT2) + own;
    float4* const T3 = reinterpret_cast<float4*>(tab + Y::oT3) + own;
    float2* const T1 = reinterpret_cast<float2*>(tab + Y::oT1) + own;
    float* const xe = tab + Y::oEdge;                         // [W][4] first (H, L), last (H, L)
    float* const xv = tab + Y::oVec;                          // [2][nv + 1]
    float* const xi = tab + Y::oInv;                          // [nv][n]
    float* const xs = tab + Y::oSp;                           // [W][2] spikes of each warp's last node
    int* const xn = reinterpret_cast<int*>(tab + Y::oInt);    // [0] PDE, [1..W] status
    double* const xd = reinterpret_cast<double*>(tab + Y::oDbl);
    const bool writer = !kUni || K == 0 || K == NL - 1;

    // slot and component of node i of the lane
    auto slot_of = [](int i) { return i == 0 ? 0 : (i < P ? P - i : i - P); };
    auto comp_of = [](int i) { return i >= P ? 1 : 0; };
    auto part = [](float4& q, int f) -> float& { return reinterpret_cast<float*>(&q)[f]; };
    auto tL = [&](int i) -> float& { return reinterpret_cast<float*>(&T1[slot_of(i) * kStride])[comp_of(i)]; };
    // 1/d and u of node i (the pivot row: 1/gamma and m_P)
    auto set_iu = [&](int i, double r, double u) {
        part(T2[slot_of(i) * kStride], comp_of(i)) = (float)r;
        part(T2[slot_of(i) * kStride], 2 + comp_of(i)) = (float)u;
    };
    // row of slot kk in the coefficient tables (uniform grids of full lanes keep slots 0, P-1)
    auto crow = [](int kk) { return kUni ? (kk == 0 ? 0 : Y::S - 1) : kk; };

    if (kPair && many_left(sh)) return;

    for (;;) {
        int pde = 0;
        if constexpr (W == 1) {
            if (k == 0) pde = atomicAdd(&counters[0], 1);
            pde = __shfl_sync(kAll, pde, 0);
        } else {
            if (K == 0) xn[0] = atomicAdd(&counters[0], 1);
            __syncthreads();
            pde = xn[0];
            __syncthreads();
        }
        if (pde >= b.m) break;
        const int N = shape_x(sh, pde), TL = shape_t(sh, pde);
        // The lane's first node.  A grid that does not fill the lanes is padded in front (negative
        // nodes, rows of the identity), so that the last node, which has no floor, is always the last
        // lane's last.
        const int j0 = kUni ? K * M : K * M - (NL * M - N);

        // ------------------------------------------------------------ setup (FP64)
        // Bound by the FP64 unit and, for few PDEs, by its latency: reciprocals by one cubic
        // Newton step, sinh and (on uniform grids) exp carried from node to node, every
        // node visited once, the lane's two halves walked at the same time.
        const double t = b.t[pde], z = b.z[pde], rr = b.r[pde], qq = b.q[pde];
        const int8_t w = b.w[pde];
        const bool amer = b.e[pde] != 0;
        const bool bad = !(t > 0.) || !(z > 0.) || !isfinite(t) || !isfinite(z) || !isfinite(rr) || !isfinite(qq);
        const Coef a = pde_coef(rr, qq, z);
        const double dt = time_step(t, TL), tdt = mul(kPair ? 0.5 : sh.theta, dt), gamma = mul(tdt, a.a0);
        const double ax_t = mul(tdt, a.ax), axx_t = mul(mul(2., tdt), a.axx);
        const double xend = mul(mul(sh.scale, z), sqrt(t));  // the grid is [-xend, xend]
        const double dy = dvd(2., (double)(N - 1));
        bool fit = !kPair || !pair64_leaves(t, z, rr, qq, w, sh.scale);
        // x_j = d sinh(y_j), y_j = yend (j dy - 1), or y_j itself on a uniform grid
        const bool uniform = kUni || sh.uniform;
        const double yend = uniform ? xend : asinh(dvd(xend, sh.density));
        const double step = mul(yend, dy);
        const double iu_u = rcp(step), im_u = mul(0.5, iu_u);
        // A walk over consecutive nodes.  Sinh grids: sinh and cosh of y_j by the addition
        // formula, with the spacing d (sinh y_(j+1) - sinh y_j) free of cancellation; where
        // the step is coarse a walk would carry the rounding of large values to the middle of
        // the grid, and every node is evaluated.  Uniform grids: s = y_j.
        struct Walk {
            double s, c, dx;  // dx: the spacing just crossed
        };
        double s1_ = 0., c1_ = 0.;  // sinh(step), cosh(step) - 1; or e^step, e^-step
        if (uniform) {
            s1_ = exp(step);
            c1_ = rcp(s1_);
        } else {
            const double h = sinh(mul(0.5, step));
            s1_ = mul(mul(2., h), sqrt(fma(h, h, 1.)));
            c1_ = mul(mul(2., h), h);
        }
        auto y_at = [&](int j) { return fma((double)j, step, -yend); };
        auto walk_at = [&](int j) -> Walk {
            const double y = y_at(j);
            if (uniform) return {y, 0., step};
            const double sy = sinh(y);
            return {sy, sqrt(fma(sy, sy, 1.)), 0.};
        };
        const bool coarse = step > 0.125;
        auto up = [&](const Walk& v, int j) -> Walk {  // to node j from j - 1
            if (uniform) return {y_at(j), 0., step};
            if (coarse) {
                const double sy = sinh(y_at(j));
                return {sy, 0., mul(sh.density, sub(sy, v.s))};
            }
            const double ds = fma(v.s, c1_, mul(v.c, s1_));
            return {add(v.s, ds), add(v.c, fma(v.c, c1_, mul(v.s, s1_))), mul(sh.density, ds)};
        };
        auto down = [&](const Walk& v, int j) -> Walk {  // to node j from j + 1
            if (uniform) return {y_at(j), 0., step};
            if (coarse) {
                const double sy = sinh(y_at(j));
                return {sy, 0., mul(sh.density, sub(v.s, sy))};
            }
            const double ds = fma(v.s, c1_, -mul(v.c, s1_));
            return {add(v.s, ds), add(v.c, fma(v.c, c1_, -mul(v.s, s1_))), -mul(sh.density, ds)};
        };
        auto x_of = [&](const Walk& v) { return uniform ? v.s : mul(sh.density, v.s); };
        auto alpha_of = [&](int j, double iu, double im) {
            return j == 0 ? mul(ax_t, iu) : (j < 0 || j >= N - 1) ? 0. : mul(im, fma(axx_t, iu, ax_t));
        };
        auto beta_of = [&](int j, double im, double id) {
            return j == N - 1 ? -mul(ax_t, id) : j <= 0 ? 0. : mul(im, fma(axx_t, id, -ax_t));
        };
        // Payoff and coefficients of node i go to the tables.  The slot's differences are D_s
        // (towards the pivot) and D_(s+1) (away from it): node a = P-k takes alpha D_s - beta
        // D_(s+1), node b = P+k beta D_s - alpha D_(s+1); slot 0 takes (alpha_0, -alpha_P) and
        // (beta_0, beta_P).
        struct Inc {
            float c1, c2, c3;
        };
        auto increments = [&](int j, double iu, double im, double id) -> Inc {
            const double ax_d = mul(dt, a.ax), axx_d = mul(mul(2., dt), a.axx);
            if (j < 0) return {0.f, 0.f, 0.f};
            if (j == 0) return {0.f, (float)mul(ax_d, iu), 0.f};
            if (j == N - 1) return {0.f, 0.f, (float)mul(ax_d, id)};
            const double drift = mul(ax_d, im), lower = mul(mul(axx_d, id), im);
            return {(float)lower, (float)add(fma(mul(axx_d, iu), im, -lower), drift), (float)drift};
        };
        auto store_coef = [&](int i, double al, double be, double iu, double im, double id) {
            const int j = j0 + i, s = slot_of(i), c = comp_of(i), r = crow(s);
            if constexpr (kPair) {
                const Split sa = split(al), sb = split(be);
                const bool swap = c == 1 && i != P;
                const float sg = i == P ? -1.f : 1.f;
                part(Cht[r * NL], c) = swap ? sb.h : sg * sa.h;
                part(Cht[r * NL], 2 + c) = swap ? sa.h : sb.h;
                part(Clt[r * NL], c) = swap ? sb.l : sg * sa.l;
                part(Clt[r * NL], 2 + c) = swap ? sa.l : sb.l;
            } else {
                // the increments' right-hand side c1 S + c2 D+ + c3 D- + c4 V (S = D+ - D-)
                const Inc q = increments(j, iu, im, id);
                const bool swap = c == 1 && i != P;
                part(Cht[r * NL], c) = i == P ? -q.c2 : swap ? -q.c3 : q.c2;
                part(Cht[r * NL], 2 + c) = i == P ? q.c3 : swap ? -q.c2 : q.c3;
                reinterpret_cast<float*>(&C1t[r * NL])[c] = q.c1;
            }
            if (kPair) fit = fit && fabs(al) < kMaxValue && fabs(be) < kMaxValue;
        };
        const double sw = w < 0 ? -1. : 1.;
        auto payoff = [&](double ex) { return split(fmax(0., fma(sw, ex, -sw))); };
        if (uniform) {
            // from the pivot outwards, e^x carried from node to node
            auto real = [&](int i, const Split& p) { return kUni || j0 + i >= 0 ? p : Split{0.f, 0.f}; };
            const double eP = exp(y_at(j0 + P));
            double ea = eP, eb = eP;
#pragma unroll 1
            for (int kk = 1; kk < P; ++kk) {
                ea = mul(ea, c1_);
                eb = mul(eb, s1_);
                const Split pa = real(P - kk, payoff(ea)), pb = real(P + kk, payoff(eb));
                PPt[kk * NL] = make_float4(pa.h, pb.h, pa.l, pb.l);
            }
            const Split p0 = real(0, payoff(mul(ea, c1_))), pP = real(P, payoff(eP));
            PPt[0] = make_float4(p0.h, pP.h, p0.l, pP.l);
        }
        auto store = [&](int i, double x, double al, double be, double iu, double im, double id) {
            const int j = j0 + i, s = slot_of(i), c = comp_of(i);
            if (!uniform) {
                const Split p = j >= 0 && ((w < 0) ? (x < 0.) : (x > 0.)) ? payoff(exp(x)) : Split{0.f, 0.f};
                part(PPt[s * NL], c) = p.h;
                part(PPt[s * NL], 2 + c) = p.l;
            }
            if (!kUni || i == 0 || i == P || i == 1 || i == M - 1) store_coef(i, al, be, iu, im, id);
        };
        // Rows of B: bl = -beta, b = 1 + alpha + beta - gamma, bu = -alpha.  The interior block
        // is eliminated from both ends: l, 1/d, u = bu/d above the pivot, m, 1/e, bl/e below.
        // The separator system needs the ends of the spikes L = B_I^-1 (bl_1 e_1) and
        // R = B_I^-1 (bu_(M-1) e_(M-1)) in FP64 (it nearly cancels on fine grids).
        double b_sep = 1., bl_sep = 0., bu_sep = 0., bl_first = 0., bu_last = 0.;
        double L1 = 0., Llast = 0., R1 = 0., Rlast = 0.;
        if constexpr (kUni && P > 1) {
            // Constant rows: the chains from both ends of a lane are the same, 1/d_k with
            // d_(k+1) = b - a c / d_k (a = bl, c = bu), and so are the spikes' sums up to
            // factors; only the last lane's descending chain differs, by its first row.  That lane
            // runs its own chain and takes the ascending one's results from lane 0.  17 FP64
            // operations per node instead of 42: 8192 PDEs of 1024 nodes set up in 0.44 ms instead of
            // 0.78 (pair arithmetic; 0.50 instead of 0.79 in FP32 stepping, 22 and 84 steps' worth).
            const bool first = K == 0, end = K == NL - 1;
            const double al = alpha_of(1, iu_u, im_u), be = beta_of(1, im_u, iu_u), edge = mul(ax_t, iu_u);
            const double ca = -be, cc = -al, cb = sub(add(1., add(al, be)), gamma);
            const double al0 = first ? edge : al, be0 = first ? 0. : be;
            bl_sep = -be0;
            bu_sep = -al0;
            b_sep = sub(add(1., add(al0, be0)), gamma);
            bl_first = ca;
            bu_last = end ? 0. : cc;
            store_coef(0, al0, be0, iu_u, im_u, iu_u);
            store_coef(P, al, be, iu_u, im_u, iu_u);
            store_coef(1, al, be, iu_u, im_u, iu_u);
            store_coef(M - 1, end ? 0. : al, end ? -edge : be, iu_u, im_u, iu_u);
            // the chain
            double r = 0., ar = 0., cr = 0., A = 1., C = 1., sig = 0.;
            double d = end ? sub(add(1., -edge), gamma) : cb, link = end ? edge : ca;
#pragma unroll 1
            for (int kk = P - 1; kk >= 1; --kk) {
                const float l = (float)ar, m = (float)cr;
                r = rcp(d);
                fit = fit && isfinite(r);
                ar = mul(link, r);
                cr = mul(cc, r);
                d = fma(-mul(cc, link), r, cb);
                sig = fma(mul(A, C), r, sig);
                A = mul(A, ar);
                C = mul(C, cr);
                const float rf = (float)r, af = (float)ar, cf = (float)cr;
                if (first) {
                    T1[kk * kStride] = f2(l, m);
                    T2[kk * kStride] = make_float4(rf, rf, cf, af);
                    T1[kk * kStride + 1].x = l;
                    T2[kk * kStride + 1].x = rf;
                    T2[kk * kStride + 1].z = cf;
                } else if (end) {
                    T1[kk * kStride].y = m;
                    T2[kk * kStride].y = rf;
                    T2[kk * kStride].w = af;
                }
                if (kk > 1) link = ca;
            }
            const double mP = cr;  // bu / d of the descending chain
            {
                const double A_ = __shfl_sync(kAll, A, 0), C_ = __shfl_sync(kAll, C, 0), s_ = __shfl_sync(kAll, sig, 0),
                             l_ = __shfl_sync(kAll, ar, 0), d_ = __shfl_sync(kAll, d, 0);
                if (end) {
                    A = A_;
                    C = C_;
                    sig = s_;
                    ar = l_;
                    d = d_;
                }
            }
            const double ig = rcp(fma(-mP, link, d));
            fit = fit && isfinite(ig);
            if (writer) {
                tL(P) = (float)ar;
                set_iu(P, ig, mP);
            }
            const double xl = -mul(mul(ca, A), ig), xr = end ? 0. : -mul(mul(cc, C), ig);
            L1 = fma(-C, xl, mul(ca, sig));
            R1 = -mul(C, xr);
            Llast = -mul(A, xl);
            Rlast = end ? 0. : fma(-A, xr, mul(cc, sig));
            if constexpr (W == 1) __syncwarp();
            else __syncthreads();
        } else {
            Walk wa = up(walk_at(j0 - 1), j0), wd = down(walk_at(j0 + M), j0 + M - 1);
            // the spacings behind each walk and their reciprocals
            double da = wa.dx, dd = wd.dx, ida = uniform ? iu_u : rcp(da), iud = uniform ? iu_u : rcp(dd);
            // ascending: 1/d, bu, products of the l and of the u, sum; descending likewise.  A row takes
            // bl bu / d of the row before it, the same product in either direction, and the first
            // row's coupling comes in at the end, so that constant rows give what the chain
            // above does, bit for bit.
            double idp = 1., bup = 0., fa = 1., pua = 1., suma = 0.;
            double iep = 1., blp = 0., fd = 1., pud = 1., sumd = 0.;
            double bP = 1., buP = 0., lP = 0.;
#pragma unroll 1
            for (int i = 0; i <= P; ++i) {
                {
                    const int j = j0 + i;
                    const Walk wn = up(wa, j + 1);
                    double iu = iu_u, im = im_u;
                    if (!uniform) {
                        iu = rcp(wn.dx);
                        im = rcp(add(wn.dx, da));
                    }
                    double al = 0., be = 0., bb = 1.;
                    if (j >= 0) {
                        al = alpha_of(j, iu, im);
                        be = beta_of(j, im, ida);
                        bb = sub(add(1., add(al, be)), gamma);
                    }
                    store(i, x_of(wa), al, be, iu, im, ida);
                    if (i == 0) {
                        bl_sep = -be;
                        b_sep = bb;
                        bu_sep = -al;
                    } else {
                        if (i == 1) bl_first = -be;
                        const double l = i == 1 ? 0. : -mul(be, idp);
                        const double d = fma(mul(be, bup), idp, bb);
                        if (i > 1) fa = mul(l, fa);
                        if (i < P) {
                            const double r = rcp(d), u = -mul(al, r);
                            fit = fit && isfinite(r);
                            if (writer) {
                                tL(i) = (float)l;
                                set_iu(i, r, u);
                            }
                            suma = fma(mul(pua, fa), r, suma);
                            pua = mul(pua, u);
                            idp = r;
                            bup = -al;
                        } else {
                            bP = d;
                            buP = -al;
                            lP = l;
                        }
                    }
                    da = wn.dx;
                    wa = wn;
                    ida = iu;
                }
                if (i > 0 && i < P) {
                    const int id_ = M - i, j = j0 + id_;
                    const Walk wn = down(wd, j - 1);
                    double idn = iu_u, im = im_u;
                    if (!uniform) {
                        idn = rcp(wn.dx);
                        im = rcp(add(wn.dx, dd));
                    }
                    double al = 0., be = 0., bb = 1.;
                    if (j >= 0) {
                        al = alpha_of(j, iud, im);
                        be = beta_of(j, im, idn);
                        bb = sub(add(1., add(al, be)), gamma);
                    }
                    store(id_, x_of(wd), al, be, iud, im, idn);
                    if (i == 1) bu_last = -al;
                    const double m = i == 1 ? 0. : -mul(al, iep);
                    const double r = rcp(fma(mul(al, blp), iep, bb)), u = -mul(be, r);
                    fit = fit && isfinite(r);
                    if (i > 1) fd = mul(m, fd);
                    if (writer) {
                        tL(id_) = (float)m;
                        set_iu(id_, r, u);
                    }
                    sumd = fma(mul(pud, fd), r, sumd);
                    pud = mul(pud, u);
                    iep = r;
                    blp = -be;
                    dd = wn.dx;
                    wd = wn;
                    iud = idn;
                }
            }
            // the pivot row (the only interior row when P = 1)
            const double mP = P > 1 ? mul(buP, iep) : 0.;
            const double ig = rcp(fma(-mP, blp, bP));
            fit = fit && isfinite(ig);
            if (P == 1) bu_last = buP;
            if (P > 1) fd = mul(mP, fd);
            if (writer) {
                tL(P) = (float)lP;
                set_iu(P, ig, mP);
            }
            // the spikes at the pivot; P - 1 sign changes, P even or 1
            const double sg = P > 1 ? -1. : 1.;
            const double xl = sg * mul(mul(bl_first, fa), ig), xr = sg * mul(mul(bu_last, fd), ig);
            L1 = fma(sg * pua, xl, mul(bl_first, suma));
            Llast = mul(sg * pud, xl);
            R1 = mul(sg * pua, xr);
            Rlast = fma(sg * pud, xr, mul(bu_last, sumd));
        }
        // the spikes, per lane straight into registers where they stay there (kReg)
        constexpr int P3 = kReg >= 1 ? P : 1;
        float4 r3[P3] = {};
        if (writer) {
            // spikes L = B_I^-1 (bl_1 e_1), R = B_I^-1 (bu_(M-1) e_(M-1)) by the steps' own solve
            auto spike = [&](float v1, float vn, int f) {
                // slots as in the steps; node 1 carries v1, node M-1 vn
                float2 v[P];
#pragma unroll
                for (int kk = 0; kk < P; ++kk) v[kk] = f2(0.f, 0.f);
                if (P > 1) v[P - 1] = f2(v1, vn);
                else v[0].y = v1 + vn;
                float2 F = f2(0.f, 0.f);
#pragma unroll
                for (int kk = P - 1; kk >= 1; --kk) v[kk] = F = fma2(neg(T1[kk * kStride]), F, v[kk]);
                const float4 qP = T2[0];
                const float xP = fmaf(-qP.w, F.y, fmaf(-T1[0].y, F.x, v[0].y)) * qP.y;
                float2 X = f2(xP, xP);
#pragma unroll
                for (int kk = 1; kk < P; ++kk) {
                    const float4 q = T2[kk * kStride];
                    v[kk] = X = fma2(neg(f2(q.z, q.w)), X, mul2(v[kk], f2(q.x, q.y)));
                }
#pragma unroll
                for (int kk = 0; kk < P; ++kk) {
                    const float b = kk > 0 ? v[kk].y : xP;
                    if constexpr (Y::kSpikeRegs) {
                        float4& q = r3[Y::kSpikeRegs ? kk : 0];
                        if (f == 0) {
                            q.x = v[kk].x;
                            q.y = b;
                        } else {
                            q.z = v[kk].x;
                            q.w = b;
                        }
                    } else {
                        float* const q = reinterpret_cast<float*>(&T3[kk * kStride]) + 2 * f;
                        if (kk > 0) q[0] = v[kk].x;
                        q[1] = b;
                    }
                }
            };
            spike((float)bl_first, 0.f, 0);
            spike(0.f, (float)bu_last, 1);
        }
        auto last_spike = [&] { return Y::kSpikeRegs ? r3[P3 - 1] : T3[(P - 1) * kStride]; };  // of node M-1
        // separator system: warp-local cyclic reduction (multipliers in FP32), and for W > 1
        // the responses to the neighbours' values and the inverse of the boundary system
        float ka[5], kc[5], ib, rq = 0.f, rs = 0.f;
        int levels = 0;  // of the reduction, as far as a multiplier is above kNoCoupling
        float sl_m = 0.f, sr_m = 0.f;  // W > 1: spikes of the previous lane's last node, as its owner uses them
        {
            double Lprev = __shfl_up_sync(kAll, Llast, 1), Rprev = __shfl_up_sync(kAll, Rlast, 1);
            if constexpr (W > 1) {
                if (k == 31) {
                    xd[2 * warp] = Llast;
                    xd[2 * warp + 1] = Rlast;
                }
                __syncthreads();
                if (k == 0 && warp > 0) {
                    Lprev = xd[2 * (warp - 1)];
                    Rprev = xd[2 * (warp - 1) + 1];
                }
            }
            if (K == 0) Lprev = Rprev = 0.;
            double al = -bl_sep * Lprev, be = b_sep - bl_sep * Rprev - bu_sep * L1, ga = -bu_sep * R1;
            // right-hand sides of the responses: -bl e_first (to ylp - Lprev s_left), ga e_last
            double vq = (W > 1 && k == 0 && warp > 0) ? -bl_sep : 0., vs = (W > 1 && k == 31 && warp < W - 1) ? ga : 0.;
            if (k == 0) al = 0.;
            if (k == 31) ga = 0.;
#pragma unroll
            for (int lv = 0; lv < 5; ++lv) {
                const int sg = 1 << lv;
                const double rb = rcp(be);
                double alm = __shfl_up_sync(kAll, al, sg), rbm = __shfl_up_sync(kAll, rb, sg),
                       gam = __shfl_up_sync(kAll, ga, sg);
                double alp = __shfl_down_sync(kAll, al, sg), rbp = __shfl_down_sync(kAll, rb, sg),
                       gap = __shfl_down_sync(kAll, ga, sg);
                if (k - sg < 0) alm = gam = 0.;
                if (k + sg > 31) alp = gap = 0.;
                const double ma = (k - sg < 0) ? 0. : mul(al, rbm), mc = (k + sg > 31) ? 0. : mul(ga, rbp);
                ka[lv] = (float)ma;
                kc[lv] = (float)mc;
                if (kCut && __any_sync(kAll, !(fabsf(ka[lv]) <= kNoCoupling && fabsf(kc[lv]) <= kNoCoupling))) levels = lv + 1;
                if constexpr (W > 1) {
                    const double qm = __shfl_up_sync(kAll, vq, sg), qp = __shfl_down_sync(kAll, vq, sg);
                    const double sm = __shfl_up_sync(kAll, vs, sg), sp = __shfl_down_sync(kAll, vs, sg);
                    vq = vq - ma * qm - mc * qp;
                    vs = vs - ma * sm - mc * sp;
                }
                be = be - ma * gam - mc * alp;
                al = -ma * alm;
                ga = -mc * gap;
            }
            const double ibd = rcp(be);
            fit = fit && isfinite(ibd);
            ib = (float)ibd;
            if constexpr (W > 1) {
                vq *= ibd;
                vs *= ibd;
                rq = (float)vq;
                rs = (float)vs;
                double* const e = xd + 2 * W;  // [W][5]: first and last responses, Lprev
                if (k == 0) {
                    e[5 * warp] = vq;
                    e[5 * warp + 1] = vs;
                    e[5 * warp + 4] = Lprev;
                }
                if (k == 31) {
                    e[5 * warp + 2] = vq;
                    e[5 * warp + 3] = vs;
                    const float4 q = last_spike();
                    xs[2 * warp] = q.y;
                    xs[2 * warp + 1] = q.w;
                }
                __syncthreads();
                if (k == 0 && warp > 0) {
                    sl_m = xs[2 * (warp - 1)];
                    sr_m = xs[2 * (warp - 1) + 1];
                }
                // boundary unknowns x_(2w) = s of warp w's last lane, x_(2w+1) = of warp w+1's
                // first: block w is [[1, h], [g, 1]], coupled to its neighbours by one entry
                // each.  Lane c of warp 0 solves for input c: the 2(W-1) local values, then
                // the W-1 values y_w of the nodes before a warp's first separator.
                if (warp == 0 && k < Y::nv) {
                    double inv00[W], inv01[W], inv10[W], inv11[W], rb[W], ra[W], up[W];
#pragma unroll
                    for (int v = 0; v < W - 1; ++v) {
                        const double q31 = e[5 * v + 2], h31 = e[5 * v + 3], lp = v > 0 ? e[5 * v + 4] : 0.;
                        const double q0 = e[5 * (v + 1)], h0 = e[5 * (v + 1) + 1], lp1 = e[5 * (v + 1) + 4];
                        double m01 = h31, m10 = q0 * lp1;
                        const double lo = q31 * lp;
                        rb[v] = k == 2 * v ? 1. : (k >= Y::n && k - Y::n + 1 == v) ? q31 : 0.;
                        ra[v] = k == 2 * v + 1 ? 1. : (k >= Y::n && k - Y::n == v) ? q0 : 0.;
                        up[v] = v + 1 < W - 1 ? h0 : 0.;
                        if (v > 0) {
                            m01 -= lo * inv01[v - 1] * up[v - 1];
                            rb[v] -= lo * (inv00[v - 1] * rb[v - 1] + inv01[v - 1] * ra[v - 1]);
                        }
                        const double det = rcp(1. - m01 * m10);
                        inv00[v] = det;
                        inv01[v] = -m01 * det;
                        inv10[v] = -m10 * det;
                        inv11[v] = det;
                    }
                    double xa = 0.;
#pragma unroll
                    for (int v = W - 2; v >= 0; --v) {
                        const double rav = ra[v] - up[v] * xa;
                        const double xb = inv00[v] * rb[v] + inv01[v] * rav;
                        xa = inv10[v] * rb[v] + inv11[v] * rav;
                        xi[k * Y::n + 2 * v] = (float)xb;
                        xi[k * Y::n + 2 * v + 1] = (float)xa;
                    }
                }
            }
        }
        const float blf = (float)bl_sep, buf = (float)bu_sep;
        bool run = __all_sync(kAll, fit) && !bad;
        if constexpr (W > 1) run = __syncthreads_and(run) != 0;
        else __syncwarp();
        if constexpr (W > 1) {
            const float4 q = last_spike();
            const float l = __shfl_up_sync(kAll, q.y, 1), r = __shfl_up_sync(kAll, q.w, 1);
            if (k > 0) {
                sl_m = l;
                sr_m = r;
            }
        }
        const float sl0 = W > 1 ? __shfl_sync(kAll, sl_m, 0) : 0.f;

        // ------------------------------------------------------------ time steps
        float2 H[P], L[P];
#pragma unroll
        for (int kk = 0; kk < P; ++kk) {
            const float4 p = PPt[kk * NL];
            H[kk] = f2(p.x, p.y);
            L[kk] = f2(p.z, p.w);
        }
        if constexpr (kPair)
            if (K == NL - 1) PPt[(P - 1) * NL].y = -INFINITY;  // the last node has no floor
        // V = max(V, p) on slot kk; in FP32 stepping X = max(X, 0)
        auto floor_at = [&](int kk, float2& h, float2& l) {
            if constexpr (kPair) {
                const float4 p = PPt[kk * NL];
                floor_to(f2(p.x, p.y), f2(p.z, p.w), h, l);
            } else {
                if (h.x < 0.f) h.x = l.x = 0.f;
                if (h.y < 0.f && (kk < P - 1 || K < NL - 1)) h.y = l.y = 0.f;  // not on the last node
            }
        };
        // the multiplier of V itself; uniform grids of full lanes: the interior multipliers
        const Split gs = split(kPair ? gamma : mul(dt, a.a0));
        const float2 gh = f2(gs.h, gs.h), gl = f2(gs.l, gs.l);
        float2 cAh{}, cAl{}, cBh{}, cBl{};
        if constexpr (kUni && kPair) {
            const double al = alpha_of(1, iu_u, im_u), be = beta_of(1, im_u, iu_u);
            const Split sa = split(al), sb = split(be);
            cAh = f2(sa.h, sb.h);
            cAl = f2(sa.l, sb.l);
            cBh = f2(sb.h, sa.h);
            cBl = f2(sb.l, sa.l);
        } else if constexpr (kUni) {
            const Inc q = increments(1, iu_u, im_u, iu_u);
            cAh = f2(q.c2, -q.c3);
            cBh = f2(q.c3, -q.c2);
            cAl = f2(q.c1, q.c1);
        }
        auto coef_h = [&](int kk, float2& A, float2& B) {
            if (kUni && kk > 0 && kk < P - 1) {
                A = cAh;
                B = cBh;
            } else {
                const float4 q = Cht[crow(kk) * NL];
                A = f2(q.x, q.y);
                B = f2(q.z, q.w);
            }
        };
        auto coef_l = [&](int kk, float2& A, float2& B) {
            if (kUni && kk > 0 && kk < P - 1) {
                A = cAl;
                B = cBl;
            } else {
                const float4 q = Clt[crow(kk) * NL];
                A = f2(q.x, q.y);
                B = f2(q.z, q.w);
            }
        };
        auto coef_s = [&](int kk) { return kUni && kk > 0 && kk < P - 1 ? cAl : C1t[crow(kk) * NL]; };
        // State of the nodes beside the lane's, -1 and M.  With one warp per PDE it comes from
        // the neighbours at the start of a step; with more, that would be one more barrier per step, so
        // every lane steps these two nodes as well, by the operations of their owners.  FP32
        // stepping: 128 PDEs of 512 nodes 0.240 -> 0.204 ms, 4096 of 2048 7.49 -> 7.09; pair arithmetic: 12
        // PDEs of 512 nodes 0.452 -> 0.430 (0.404 since solve() gives the neighbour's value without
        // waiting for its owner), but 4096 of 2048 uniform nodes 6.21 -> 6.46, where the two
        // nodes cost more than the barrier (kOwn).
        float2 Hn, Ln;
        auto neighbours = [&]() {
            const float2 last = P > 1 ? f2(H[P - 1].y, L[P - 1].y) : f2(H[0].y, L[0].y);
            Hn = f2(__shfl_up_sync(kAll, last.x, 1), __shfl_down_sync(kAll, H[0].x, 1));
            Ln = f2(__shfl_up_sync(kAll, last.y, 1), __shfl_down_sync(kAll, L[0].x, 1));
            if constexpr (W > 1) {
                if (k == 0) {
                    xe[4 * warp] = H[0].x;
                    xe[4 * warp + 1] = L[0].x;
                }
                if (k == 31) {
                    xe[4 * warp + 2] = last.x;
                    xe[4 * warp + 3] = last.y;
                }
                __syncthreads();
                if (k == 0 && warp > 0) {
                    Hn.x = xe[4 * warp - 2];
                    Ln.x = xe[4 * warp - 1];
                }
                if (k == 31 && warp < W - 1) {
                    Hn.y = xe[4 * warp + 4];
                    Ln.y = xe[4 * warp + 5];
                }
            }
            if (K == 0) Hn.x = Ln.x = 0.f;
            if (K == NL - 1) Hn.y = Ln.y = 0.f;
        };

        // FP32 stepping carries X = V - p (fd1d_fp32.cu).  X starts at zero; the payoff waits in
        // the result row, and its tables give way to the constant part q = dt A p of the
        // residual, from pair arithmetic with the steps' own rounded coefficients.  FP32 cannot
        // hold q at the payoff's kink, and the same rounding every step would triple the
        // error (grid of 2048 nodes, density 0.25: 1.1e-9 to 6e-9); passed on to the next node, where q is
        // small, it moves by a node instead (1.0e-9).
        float2* const qt = reinterpret_cast<float2*>(tab + Y::oPP) + K;
        float2 q_low{};
        double* const V = vout + shape_row(sh, pde);
        if (!kPair && run) {
            neighbours();
            auto payoff = [&](int kk) {
                const float4 p = PPt[kk * NL];
                return PP2{f2(p.x, p.y), f2(p.z, p.w)};
            };
            // q of slot kk over its payoffs; V = p
            auto source = [&](int kk, const PP2& p, const PP2& X, const PP2& Z, const PP2& S) {
                float2 A, B, low = f2(0.f, 0.f), s1, s2, s, e;
                coef_h(kk, A, B);
                auto product = [&](float2 a, const PP2& v) {
                    const float2 t = mul2(a, v.h);
                    low = add2(low, fma2(a, v.l, fma2(a, v.h, neg(t))));
                    return t;
                };
                const float2 tS = product(coef_s(kk), S), tX = product(A, X), tZ = product(B, Z), tV = product(gh, p);
                two_sum(tS, tX, s1, e);
                low = add2(low, e);
                two_sum(tZ, tV, s2, e);
                low = add2(low, e);
                two_sum(s1, s2, s, e);
                low = add2(low, e);
                const float2 h = add2(s, low), l = sub2(low, sub2(h, s));
                PPt[kk * NL] = make_float4(h.x, h.y, l.x, l.y);
                const int na = j0 + (kk == 0 ? 0 : P - kk), nb = j0 + P + kk;
                if (na >= 0) V[na] = (double)p.h.x + (double)p.l.x;
                if (nb >= 0) V[nb] = (double)p.h.y + (double)p.l.y;
            };
            const PP2 p0 = payoff(0);
            PP2 c = {f2(p0.h.y, p0.h.y), f2(p0.l.y, p0.l.y)}, Dc{}, D1{};
#pragma unroll 1
            for (int kk = 1; kk <= P; ++kk) {
                const PP2 next = kk < P ? payoff(kk) : PP2{f2(p0.h.x, Hn.y), f2(p0.l.x, Ln.y)};
                const PP2 Dn = pair_diff(c, next);
                if (kk == 1) D1 = Dn;
                else source(kk - 1, c, Dc, Dn, pair_diff(Dc, Dn));
                Dc = Dn;
                c = next;
            }
            const PP2 E = pair_diff(p0, {f2(Hn.x, 0.f), f2(Ln.x, 0.f)});
            const PP2 X = {f2(Dc.h.x, D1.h.y), f2(Dc.l.x, D1.l.y)}, Z = {f2(E.h.x, D1.h.x), f2(E.l.x, D1.l.x)};
            source(0, p0, X, Z, pair_diff({f2(X.h.x, -X.h.y), f2(X.l.x, -X.l.y)}, Z));
            // lo to the next node, from both ends of the lane to the pivot
#pragma unroll
            for (int kk = 0; kk < P; ++kk) {
                const PP2 v = payoff(kk);
                H[kk] = v.h;
                L[kk] = v.l;
            }
            if constexpr (P > 1) {
                float2 rest = f2(L[0].x, 0.f);
#pragma unroll
                for (int kk = P - 1; kk >= 1; --kk) {
                    const float2 l = add2(rest, L[kk]), h = add2(H[kk], l);
                    rest = sub2(l, sub2(h, H[kk]));
                    H[kk] = h;
                }
                const float lP = (rest.x + rest.y) + L[0].y, hP = H[0].y + lP;
                const float last = lP - (hP - H[0].y);
                H[0].y = hP;
                if (fabsf(H[1].x) < fabsf(H[1].y)) H[1].x += last;
                else H[1].y += last;
            } else {
                q_low = L[0];  // two nodes a lane: both may lie at the kink
            }
            if constexpr (W == 1) __syncwarp();
            else __syncthreads();
#pragma unroll
            for (int kk = 0; kk < P; ++kk) {
                qt[kk * NL] = H[kk];
                H[kk] = L[kk] = f2(0.f, 0.f);
            }
            Hn = Ln = f2(0.f, 0.f);
        }
        if (kPair && kOwn && run) neighbours();
        const float2 pHn = Hn, pLn = Ln;  // pairs: the payoffs at the two nodes

        // factors held in registers for the whole PDE (kReg)
        constexpr int P1 = kReg >= 3 ? P : 1, P2 = kReg >= 2 ? P : 1;
        float2 r1[P1];
        float4 r2[P2];
#pragma unroll
        for (int kk = 0; kk < P1; ++kk) r1[kk] = T1[kk * kStride];
#pragma unroll
        for (int kk = 0; kk < P2; ++kk) r2[kk] = T2[kk * kStride];
        if constexpr (!Y::kSpikeRegs) {
#pragma unroll
            for (int kk = 0; kk < P3; ++kk) r3[kk] = T3[kk * kStride];
        }
        auto fac1 = [&](int kk) -> float2 { return kReg >= 3 ? r1[kReg >= 3 ? kk : 0] : T1[kk * kStride]; };
        auto fac2 = [&](int kk) -> float4 { return kReg >= 2 ? r2[kReg >= 2 ? kk : 0] : T2[kk * kStride]; };
        auto fac3 = [&](int kk) -> float4 { return kReg >= 1 ? r3[kReg >= 1 ? kk : 0] : T3[kk * kStride]; };
        // B x = y in FP32, in place on the slots; s1: x of the next lane's separator, um: x of
        // the previous lane's last node
        auto solve = [&](float2 (&y)[P], int which, float& s1, float& um) {
            phase_edge<kEdge>();
            float2 F = f2(0.f, 0.f);
#pragma unroll
            for (int kk = P - 1; kk >= 1; --kk) {
                F = fma2(neg(fac1(kk)), F, y[kk]);
                y[kk] = F;
            }
            const float4 p2 = fac2(0), p3 = fac3(0);
            const float yP = fmaf(-p2.w, F.y, fmaf(-fac1(0).y, F.x, y[0].y)) * p2.y;
            float2 X = f2(yP, yP);
#pragma unroll
            for (int kk = 1; kk < P; ++kk) {
                const float4 q = fac2(kk);
                X = fma2(neg(f2(q.z, q.w)), X, mul2(y[kk], f2(q.x, q.y)));
                y[kk] = X;
            }
            const float y_last = X.y, y_first = X.x;  // nodes M-1 and 1 (the pivot when P = 1)
            float ylp = __shfl_up_sync(kAll, y_last, 1);
            if (k == 0) ylp = 0.f;
            float rho = fmaf(-buf, y_first, fmaf(-blf, ylp, y[0].x));
#pragma unroll
            for (int lv = 0; lv < 5; ++lv) {
                if (kCut && lv >= levels) break;
                const float rm = __shfl_up_sync(kAll, rho, 1 << lv), rp = __shfl_down_sync(kAll, rho, 1 << lv);
                rho = fmaf(-kc[lv], rp, fmaf(-ka[lv], rm, rho));
            }
            float s = rho * ib;
            if constexpr (W == 1) {
                s1 = __shfl_down_sync(kAll, s, 1);
                if (k == 31) s1 = 0.f;
                phase_edge<kEdge>();
            } else {
                // inputs: z of the warp boundaries, then y of the nodes before each warp
                float* const v = xv + which * (Y::nv + 1);
                if (k == 31 && warp < W - 1) {
                    v[2 * warp] = s;
                    v[Y::n + warp] = y_last;
                }
                if (k == 0 && warp > 0) v[2 * warp - 1] = s;
                __syncthreads();
                const int row = k < Y::n ? k : 0;
                float x0 = 0.f, x1 = 0.f, x2 = 0.f;
#pragma unroll
                for (int c = 0; c < W - 1; ++c) {
                    x0 = fmaf(xi[(3 * c) * Y::n + row], v[3 * c], x0);
                    x1 = fmaf(xi[(3 * c + 1) * Y::n + row], v[3 * c + 1], x1);
                    x2 = fmaf(xi[(3 * c + 2) * Y::n + row], v[3 * c + 2], x2);
                }
                const float x = (x0 + x1) + x2;
                const float bl_ = __shfl_sync(kAll, x, warp > 0 ? 2 * warp - 2 : 0);       // left warp's last
                const float a_ = __shfl_sync(kAll, x, warp > 0 ? 2 * warp - 1 : 0);        // own first
                const float b_ = __shfl_sync(kAll, x, warp < W - 1 ? 2 * warp : 0);        // own last
                const float ar = __shfl_sync(kAll, x, warp < W - 1 ? 2 * warp + 1 : 0);    // right warp's first
                const float yl = warp > 0 ? v[Y::n + warp - 1] : 0.f;
                const float Q = warp > 0 ? fmaf(-sl0, bl_, yl) : 0.f, Sr = warp < W - 1 ? ar : 0.f;
                s = fmaf(-rs, Sr, fmaf(rq, Q, s));
                if (k == 0 && warp > 0) s = a_;
                if (k == 31 && warp < W - 1) s = b_;
                s1 = __shfl_down_sync(kAll, s, 1);
                if (k == 31) s1 = Sr;
                if constexpr (kPair || kOwn) {
                    // by the operations its owner uses below, without waiting for them
                    float s_prev = __shfl_up_sync(kAll, s, 1);
                    if (k == 0) {
                        s_prev = bl_;
                        ylp = yl;
                    }
                    um = fmaf(-s, sr_m, fmaf(-s_prev, sl_m, ylp));
                }
            }
            const float2 ms = f2(-s, -s), ms1 = f2(-s1, -s1);
#pragma unroll
            for (int kk = 1; kk < P; ++kk) {
                const float4 q = fac3(kk);
                y[kk] = fma2(ms1, f2(q.z, q.w), fma2(ms, f2(q.x, q.y), y[kk]));
            }
            y[0] = f2(s, fmaf(-s1, p3.w, fmaf(-s, p3.y, yP)));
            if constexpr (kPair && W == 1) {
                um = __shfl_up_sync(kAll, P > 1 ? y[P - 1].y : y[0].y, 1);
                if (K == 0) um = 0.f;
            }
        };

        if (run) {
            for (int step = 1; step < TL; ++step) {
                if constexpr (!kOwn) neighbours();
                phase_edge<kEdge>();

                // D_k = V of slot k-1 minus V of slot k (the pivot in both components before slot
                // 1, nodes 0 and M after slot P-1), high and low parts each exact
                auto diff = [&](int kk, float2& dh, float2& dl) {
                    dh = sub2(kk == 1 ? f2(H[0].y, H[0].y) : H[kk - 1], kk == P ? f2(H[0].x, Hn.y) : H[kk]);
                    dl = sub2(kk == 1 ? f2(L[0].y, L[0].y) : L[kk - 1], kk == P ? f2(L[0].x, Ln.y) : L[kk]);
                };
                float2 y[P];
                float s1, um;
                if constexpr (!kPair) {
                    // the residual dt A X + q, then X += B^-1 of it
                    float2 h1, l1;
                    diff(1, h1, l1);
                    float2 hc = h1, lc = l1, dc = add2(h1, l1);
#pragma unroll
                    for (int kk = 1; kk < P; ++kk) {
                        float2 hn, ln, A, B;
                        diff(kk + 1, hn, ln);
                        coef_h(kk, A, B);
                        const float2 dn = add2(hn, ln), S = add2(sub2(hc, hn), sub2(lc, ln));
                        const float2 r = fma2(coef_s(kk), S, fma2(gh, add2(H[kk], L[kk]), qt[kk * NL]));
                        y[kk] = fma2(B, dn, fma2(A, dc, r));
                        hc = hn;
                        lc = ln;
                        dc = dn;
                    }
                    float2 A, B;
                    coef_h(0, A, B);
                    const float eh = H[0].x - Hn.x, el = L[0].x - Ln.x;
                    const float2 S = f2((hc.x - eh) + (lc.x - el), -(h1.y + h1.x) - (l1.y + l1.x));
                    float2 r = fma2(coef_s(0), S, fma2(gh, add2(H[0], L[0]), qt[0]));
                    if constexpr (P == 1) r = add2(r, q_low);
                    y[0] = fma2(B, f2(eh + el, h1.x + l1.x), fma2(A, f2(dc.x, h1.y + l1.y), r));
                    solve(y, kOwn ? step & 1 : 0, s1, um);
                    phase_edge<kEdge>();
#pragma unroll
                    for (int kk = 0; kk < P; ++kk) {
                        ff_acc2(H[kk], L[kk], y[kk]);
                        if (amer) floor_at(kk, H[kk], L[kk]);
                    }
                    if constexpr (kOwn) {
                        ff_acc2(Hn, Ln, f2(um, s1));
                        if (amer) {
                            if (Hn.x < 0.f) Hn.x = Ln.x = 0.f;
                            if (Hn.y < 0.f) Hn.y = Ln.y = 0.f;
                        }
                    }
                } else {
                    // 1. u0 = B^-1 A' V in FP32.  D_k = V of slot k-1 minus V of slot k (the pivot
                    // in both components before slot 1, nodes 0 and M after slot P-1)
                    um = 0.f;
                    {
                        float2 Dc = f2(0.f, 0.f), D1 = f2(0.f, 0.f);
#pragma unroll
                        for (int kk = 1; kk <= P; ++kk) {
                            const float2 hu = kk == 1 ? f2(H[0].y, H[0].y) : H[kk - 1];
                            const float2 lu = kk == 1 ? f2(L[0].y, L[0].y) : L[kk - 1];
                            const float2 hd = kk == P ? f2(H[0].x, Hn.y) : H[kk];
                            const float2 ld = kk == P ? f2(L[0].x, Ln.y) : L[kk];
                            const float2 Dn = add2(sub2(hu, hd), sub2(lu, ld));
                            if (kk == 1) {
                                D1 = Dn;
                            } else {
                                float2 A, B;
                                coef_h(kk - 1, A, B);
                                y[kk - 1] = fma2(A, Dc, fma2(neg(B), Dn, mul2(gh, H[kk - 1])));
                            }
                            Dc = Dn;
                        }
                        float2 A, B;
                        coef_h(0, A, B);
                        const float E = (H[0].x - Hn.x) + (L[0].x - Ln.x);
                        y[0] = fma2(A, f2(Dc.x, D1.y), fma2(neg(B), f2(E, D1.x), mul2(gh, H[0])));
                    }
                    solve(y, 0, s1, um);

                    const float2 un = f2(um, s1);

                    // 2., 3. W = V + u0 and r = A' W - u0
                    float2 u0[P];
                    phase_edge<kEdge>();
                    {
                        const PP2 w0 = shifted(H[0], L[0], y[0]);
                        const PP2 wn = shifted(Hn, Ln, un);  // nodes -1 and M
                        PP2 wc = {f2(w0.h.y, w0.h.y), f2(w0.l.y, w0.l.y)};           // slot k-1
                        u0[0] = y[0];
                        PP2 Dc{}, D1{};
#pragma unroll
                        for (int kk = 1; kk <= P; ++kk) {
                            PP2 wk;
                            if (kk < P) {
                                wk = shifted(H[kk], L[kk], y[kk]);
                                u0[kk] = y[kk];
                            } else {
                                wk = {f2(w0.h.x, wn.h.y), f2(w0.l.x, wn.l.y)};
                            }
                            const PP2 Dn = pair_diff_norm(wc, wk);
                            if (kk == 1) {
                                D1 = Dn;
                            } else {
                                float2 Ah, Al, Bh, Bl;
                                coef_h(kk - 1, Ah, Bh);
                                coef_l(kk - 1, Al, Bl);
                                y[kk - 1] = pair_residual(Ah, Al, Dc, Bh, Bl, Dn, gh, gl, wc, u0[kk - 1]);
                            }
                            Dc = Dn;
                            wc = wk;
                        }
                        const PP2 E = pair_diff_norm(w0, {f2(wn.h.x, 0.f), f2(wn.l.x, 0.f)});
                        float2 Ah, Al, Bh, Bl;
                        coef_h(0, Ah, Bh);
                        coef_l(0, Al, Bl);
                        const PP2 X = {f2(Dc.h.x, D1.h.y), f2(Dc.l.x, D1.l.y)}, Z = {f2(E.h.x, D1.h.x), f2(E.l.x, D1.l.x)};
                        y[0] = pair_residual(Ah, Al, X, Bh, Bl, Z, gh, gl, w0, u0[0]);
                    }
                    // 4. e = B^-1 r, V' = max(V + 2 u0 + 2 e, p)
                    solve(y, 1, s1, um);
                    phase_edge<kEdge>();
#pragma unroll
                    for (int kk = 0; kk < P; ++kk) {
                        pair_acc2(H[kk], L[kk], u0[kk], y[kk]);
                        if (amer) floor_at(kk, H[kk], L[kk]);
                    }
                    if constexpr (kOwn) {
                        pair_acc2(Hn, Ln, un, f2(um, s1));
                        if (amer) floor_to(pHn, pLn, Hn, Ln);
                    }
                }
            }
        }
        // ------------------------------------------------------------ result
        bool fin = run;
        if constexpr (kPair) {
#pragma unroll
            for (int kk = 0; kk < P; ++kk) fin = fin && isfinite(H[kk].x) && isfinite(H[kk].y);
            fin = __all_sync(kAll, fin);
            if constexpr (W > 1) fin = __syncthreads_and(fin) != 0;
        }
        if (fin) {
#pragma unroll
            for (int kk = 0; kk < P; ++kk) {
                const int na = j0 + (kk == 0 ? 0 : P - kk), nb = j0 + P + kk;
                const double va = (double)H[kk].x + (double)L[kk].x, vb = (double)H[kk].y + (double)L[kk].y;
                if (na >= 0) V[na] = kPair ? va : V[na] + va;
                if (nb >= 0) V[nb] = kPair ? vb : V[nb] + vb;
            }
        }
        if (K == 0) {
            pde_status[pde] = bad ? KWG_STATUS_BAD_INPUT : run || kPair ? KWG_STATUS_OK : KWG_STATUS_SOLVER;
            if constexpr (kPair)
                if (!fin && !bad) rescue[atomicAdd(&counters[2], 1)] = pde;
        }
        // the tables are rewritten for the next PDE
        if constexpr (!kPair && W > 1) __syncthreads();
        else __syncwarp();
    }
}

namespace {

// Resident blocks per SM of a variant, set by prepare_onchip.
template <int M, bool kUni, int W, bool kPair>
int& per_sm_onchip()
{
    static int v = 1;
    return v;
}

template <int M, bool kUni, int W, bool kPair>
void prepare_onchip()
{
    constexpr size_t smem = Lay<M, kUni, W, kPair>::kBytes;
    auto kern = fd1d_solve_onchip<M, kUni, W, kPair>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * W, smem);
    per_sm_onchip<M, kUni, W, kPair>() = per_sm < 1 ? 1 : per_sm;
}

template <int M, bool kUni, int W, bool kPair>
void launch_onchip(const PdeBatch& b, const Fd1dShape& sh, double* vout, int32_t* pde_status, int* counters,
                   int32_t* rescue, int sms, cudaStream_t stream)
{
    const int cap = sms * per_sm_onchip<M, kUni, W, kPair>();
    fd1d_solve_onchip<M, kUni, W, kPair><<<b.m < cap ? b.m : cap, 32 * W, Lay<M, kUni, W, kPair>::kBytes, stream>>>(
        b, sh, vout, pde_status, counters, rescue);
}

}  // namespace

}  // namespace kwg
