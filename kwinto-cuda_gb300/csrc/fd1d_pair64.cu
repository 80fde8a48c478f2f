// fd1d_pair64.cu -- the FP64 theta-scheme solve (theta = 1/2) on the FP32 units: one to
// eight warps per PDE, the whole PDE on chip, values as pairs of floats and one step of
// iterative refinement per time step.
//
// Why.  A warp-wide FP64 instruction holds its scheduler's FP64 unit for 64 cycles, a
// warp-wide FP32 one for 1.  The streaming kernel's three FP64 multiply-adds per node-step
// (fd1d_fp64.cu) therefore cost 6 scheduler cycles per node; the ~76 FP32 operations here
// cost 2.4, and their latency is 4 cycles instead of 64.
//
// Bound by the FP32 pipe (two thirds busy at 1024 uniform nodes) and, for few PDEs, by the
// latency of the two separator solves per step.  Measured against the FP64 solvers that took
// these shapes before (whole calls): 32768 PDEs, 1024 x 1024 uniform, 192 -> 93 ms; 8192 PDEs,
// 1024 x 1024, density 0.25, 186 -> 28 ms; 777 PDEs, 1000 x 731, 12.4 -> 2.8 ms; 600 PDEs,
// 512 x 512, 2.50 -> 0.87 ms; 12 PDEs 2.35 -> 0.52 ms; 131072 uneven PDEs 339 -> 155 ms.
//
// Numerics.  The reference step B V' = E V (src/Math/kwFd1d.cpp:61-132) is taken in
// increments.  With A' = theta dt A and u = theta (V' - V) it reads
//     u = A' (V + u),       V' = max(V + 2 u, p),
// and A' in difference form,
//     (A' W)_j = alpha_j (W_{j+1} - W_j) - beta_j (W_j - W_{j-1}) + gamma W_j.
//   1. u0 = B^-1 (A' V) in FP32;
//   2. W = V + u0 as a pair;
//   3. r = A' W - u0 in pair arithmetic (error-free differences, products and sums; alpha,
//      beta and gamma as pairs): the two sides cancel to ~1e-7 V, and what is left has
//      ~2^-48 V of error;
//   4. e = B^-1 r in FP32, and V' = max(V + 2 u0 + 2 e, p) with V and p as pairs
//      (~49 significant bits, renormalised every step).
// An FP32 solve has a relative error of ~1e-7, so u0 + e has one of ~1e-14 V.  Rounding a
// tridiagonal row in FP64 perturbs V by ~1e-15 per step, always the same way; the
// difference form has no such drift.  On the 1024 x 1024 uniform grid the largest error
// against the scheme in exact arithmetic is 3e-13 relative where the FP64 sweeps have
// 2e-12 (CPU emulation over random options, |x| < 0.75).
//
// What it does not take: theta != 1/2, more than 2048 nodes, and -- PDE by PDE, found in
// the setup or at the end -- values beyond FP32's range, and grids that a drift crosses
// (|r - q - z^2/2| T above kMaxDrift half-widths), where the one-sided boundary rows of the
// scheme amplify whatever stands at the boundary by orders of magnitude.  Those PDEs go
// to a list that the FP64 kernel of fd1d_pcr64.cu works off in a launch of its own.
//
// Solve of B u = r (the partition of fd1d_fp32.cu): lane K owns nodes K M .. K M + M - 1,
// node K M is a separator, the others are eliminated from both ends towards the lane's
// pivot node P = M / 2, and the separator system is solved by cyclic reduction over the
// warp.  With W > 1 warps per PDE each warp reduces its own 32 separators, and the
// 2 (W - 1) values at the warp boundaries come from one dense product with the inverse of
// their system (one block barrier per solve instead of one per reduction level).
//
// Packed pairs.  As in fd1d_fp32.cu, nodes P-k and P+k share a float2 (slot k; slot 0 holds
// nodes 0 and P) and every step runs on packed FP32 instructions, which need half the
// issue slots of scalar ones at the same FP32 rate.
#include <cstdint>
#include <cuda_runtime.h>

#include "fd1d_common.cuh"
#include "fd1d_kernels.h"

namespace kwg {

namespace {

constexpr unsigned kAll = 0xffffffffu;
// Half-widths that the drift may cross; beyond it the boundary's growth reaches the
// middle of the grid and FP32's range no longer holds it.
constexpr double kMaxDrift = 0.3;
// Payoffs and coefficients above this leave no room for the pair arithmetic in FP32's range.
constexpr double kMaxValue = 1e30, kMaxLog = 69.;

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
// PDE no barrier stands between the phases, and the loads it moved up cost registers (M = 32:
// 255 and 444 bytes of spills without, 255 and none with).
__device__ __forceinline__ void phase_edge() { __syncwarp(); }

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

// 1 / d by Newton's method in its cubic form, r (1 + e + e^2) with e = 1 - d r, from the
// hardware's 20-bit estimate: the error left is e^3 ~ 2^-60, then rounding.  Zero and
// non-finite d give a non-finite result.
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

// Warps per SM that the registers must leave room for.  More (16 at M = 16, 20 at M = 8, 24 at
// M = 4) spills a little and is no faster: 8192 PDEs of 512 uniform nodes 6.09 ms at 12, 6.12 at 16.
constexpr int min_warps(int M) { return M == 32 ? 8 : M == 16 ? 12 : 16; }

// Shared-memory layout of one PDE group (floats).  P = M / 2 slots, NL = 32 W lanes.
//   PPt  [P][NL] float4   payoff (hi_a, hi_b, lo_a, lo_b); -inf where no floor applies
//   Cht  [S][NL] float4   (A_a, A_b, B_a, B_b) high parts, Clt low parts: the multipliers
//                         of a slot's two differences (below); S = P, or on uniform grids
//                         of full lanes the two slots that can hold a boundary node
//   T1 (l), T2 (1/d, u), T3 (spikes L, R): the factors, [P][stride]; on uniform grids of
//                         full lanes once for the group and once for the last lane
// then the exchange area of W > 1.
template <int M, bool kUni, int W>
struct Lay {
    static constexpr int P = M / 2, NL = 32 * W;
    static constexpr int S = kUni ? (P > 1 ? 2 : 1) : P;
    static constexpr int kStride = kUni ? 2 : NL;
    static constexpr int oPP = 0;
    static constexpr int oCh = oPP + 4 * P * NL;
    static constexpr int oCl = oCh + 4 * S * NL;
    static constexpr int oT2 = oCl + 4 * S * NL;
    static constexpr int oT3 = oT2 + 4 * P * kStride;
    static constexpr int oT1 = oT3 + 4 * P * kStride;
    static constexpr int oX = oT1 + 2 * P * kStride;
    static constexpr int n = 2 * (W - 1), nv = 3 * (W - 1);  // boundary unknowns and their inputs
    // exchange area: edges [W][4], inputs of the two solves [2][nv], inverse [nv][n],
    // spikes at the warp boundaries [W][2], PDE number and status
    static constexpr int oEdge = oX, oVec = oEdge + 4 * W, oInv = oVec + 2 * (nv + 1), oSp = oInv + nv * n,
                         oInt = oSp + 2 * W;
    static constexpr int kEx = W == 1 ? 0 : 4 * W + 2 * (nv + 1) + nv * n + 2 * W + W + 2;
    // setup exchange in doubles, over the payoff table's space is not possible (in use):
    // [3][W] boundary couplings, [2][W] neighbour spikes
    static constexpr int oDbl = (oX + kEx + 1) / 2 * 2;
    static constexpr int kDbl = W == 1 ? 0 : 2 * 7 * W;
    static constexpr size_t kBytes = (size_t)(oDbl + kDbl) * sizeof(float);
};

}  // namespace

template <int M, bool kUni, int W>
__global__ void __launch_bounds__(32 * W, min_warps(M) / W) fd1d_solve_pair64(const PdeBatch b, Fd1dShape sh, double* __restrict__ vout,
                                                            int32_t* __restrict__ pde_status,
                                                            int* __restrict__ counters, int32_t* __restrict__ rescue)
{
    using Y = Lay<M, kUni, W>;
    constexpr int P = Y::P, NL = Y::NL, kStride = Y::kStride;
    static_assert(M >= 2 && M % 2 == 0, "as many rows above the pivot as below");
    extern __shared__ __align__(16) float tab[];
    const int k = threadIdx.x & 31, warp = W == 1 ? 0 : threadIdx.x >> 5;
    const int K = threadIdx.x;
    const int own = kUni ? (K + 1) / NL : K;
    float4* const PPt = reinterpret_cast<float4*>(tab + Y::oPP) + K;
    float4* const Cht = reinterpret_cast<float4*>(tab + Y::oCh) + K;
    float4* const Clt = reinterpret_cast<float4*>(tab + Y::oCl) + K;
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
    auto tID = [&](int i) -> float& { return part(T2[slot_of(i) * kStride], comp_of(i)); };
    auto tU = [&](int i) -> float& { return part(T2[slot_of(i) * kStride], 2 + comp_of(i)); };
    auto tSL = [&](int i) -> float& { return part(T3[slot_of(i) * kStride], comp_of(i)); };
    auto tSR = [&](int i) -> float& { return part(T3[slot_of(i) * kStride], 2 + comp_of(i)); };
    // row of slot kk in the coefficient tables (uniform grids of full lanes keep slots 0, P-1)
    auto crow = [](int kk) { return kUni ? (kk == 0 ? 0 : Y::S - 1) : kk; };

    const int j0 = K * M;
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

        // ------------------------------------------------------------ setup (FP64)
        // Bound by the FP64 unit and, for few PDEs, by its latency: reciprocals by one cubic
        // Newton step, sinh and (on uniform grids) exp carried from node to node, every
        // node visited once, the lane's two halves walked at the same time.
        const double t = b.t[pde], z = b.z[pde], rr = b.r[pde], qq = b.q[pde];
        const int8_t w = b.w[pde];
        const bool amer = b.e[pde] != 0;
        const bool bad = !(t > 0.) || !(z > 0.) || !isfinite(t) || !isfinite(z) || !isfinite(rr) || !isfinite(qq);
        const Coef a = pde_coef(rr, qq, z);
        const double tdt = mul(0.5, time_step(t, TL)), gamma = mul(tdt, a.a0);
        const double ax_t = mul(tdt, a.ax), axx_t = mul(mul(2., tdt), a.axx);
        const double xend = mul(mul(sh.scale, z), sqrt(t));  // the grid is [-xend, xend]
        const double dy = dvd(2., (double)(N - 1));
        bool fit = fabs(a.ax) * t <= kMaxDrift * xend && (w < 0 || xend < kMaxLog);
        // x_j = d sinh(y_j), y_j = yend (j dy - 1), or y_j itself on a uniform grid
        const bool uniform = kUni || sh.uniform;
        const double yend = uniform ? xend : asinh(dvd(xend, sh.density));
        const double step = mul(yend, dy);
        const double iu_u = rcp(step), im_u = mul(0.5, iu_u);
        // A walk over consecutive nodes.  Sinh grids: sinh and cosh of y_j by the addition
        // formula, with the spacing d (sinh y_(j+1) - sinh y_j) free of cancellation; where
        // the step is coarse a walk would carry the rounding of large values to the middle of
        // the grid, and every node is evaluated.  Uniform grids: s = y_j, c = e^(y_j).
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
            if (uniform) return {y, exp(y), step};
            const double sy = sinh(y);
            return {sy, sqrt(fma(sy, sy, 1.)), 0.};
        };
        const bool coarse = step > 0.125;
        auto up = [&](const Walk& v, int j) -> Walk {  // to node j from j - 1
            if (uniform) return {y_at(j), mul(v.c, s1_), step};
            if (coarse) {
                const double sy = sinh(y_at(j));
                return {sy, 0., mul(sh.density, sub(sy, v.s))};
            }
            const double ds = fma(v.s, c1_, mul(v.c, s1_));
            return {add(v.s, ds), add(v.c, fma(v.c, c1_, mul(v.s, s1_))), mul(sh.density, ds)};
        };
        auto down = [&](const Walk& v, int j) -> Walk {  // to node j from j + 1
            if (uniform) return {y_at(j), mul(v.c, c1_), step};
            if (coarse) {
                const double sy = sinh(y_at(j));
                return {sy, 0., mul(sh.density, sub(v.s, sy))};
            }
            const double ds = fma(v.s, c1_, -mul(v.c, s1_));
            return {add(v.s, ds), add(v.c, fma(v.c, c1_, -mul(v.s, s1_))), -mul(sh.density, ds)};
        };
        auto x_of = [&](const Walk& v) { return uniform ? v.s : mul(sh.density, v.s); };
        auto alpha_of = [&](int j, double iu, double im) {
            return j == 0 ? mul(ax_t, iu) : j >= N - 1 ? 0. : mul(im, fma(axx_t, iu, ax_t));
        };
        auto beta_of = [&](int j, double im, double id) {
            return j == N - 1 ? -mul(ax_t, id) : (j == 0 || j >= N) ? 0. : mul(im, fma(axx_t, id, -ax_t));
        };
        // Payoff and coefficients of node i go to the tables.  The slot's differences are D_s
        // (towards the pivot) and D_(s+1) (away from it): node a = P-k takes alpha D_s - beta
        // D_(s+1), node b = P+k beta D_s - alpha D_(s+1); slot 0 takes (alpha_0, -alpha_P) and
        // (beta_0, beta_P).
        auto store = [&](int i, double x, double ex, double al, double be) {
            const int j = j0 + i, s = slot_of(i), c = comp_of(i);
            double p = 0.;
            if (j < N && ((w < 0) ? (x < 0.) : (x > 0.))) {
                if (!uniform) ex = exp(x);
                p = fmax(0., (w < 0) ? sub(1., ex) : sub(ex, 1.));
            }
            const Split ph = split(p);
            part(PPt[s * NL], c) = ph.h;
            part(PPt[s * NL], 2 + c) = ph.l;
            if (!kUni || i == 0 || i == P || i == 1 || i == M - 1) {
                const Split sa = split(al), sb = split(be);
                const int r = crow(s);
                const bool swap = c == 1 && i != P;
                const float sg = i == P ? -1.f : 1.f;
                part(Cht[r * NL], c) = swap ? sb.h : sg * sa.h;
                part(Cht[r * NL], 2 + c) = swap ? sa.h : sb.h;
                part(Clt[r * NL], c) = swap ? sb.l : sg * sa.l;
                part(Clt[r * NL], 2 + c) = swap ? sa.l : sb.l;
            }
            fit = fit && fabs(al) < kMaxValue && fabs(be) < kMaxValue;
        };
        // Rows of B: bl = -beta, b = 1 + alpha + beta - gamma, bu = -alpha.  The interior block
        // is eliminated from both ends: l, 1/d, u = bu/d above the pivot, m, 1/e, bl/e below.
        // The separator system needs the ends of the spikes L = B_I^-1 (bl_1 e_1) and
        // R = B_I^-1 (bu_(M-1) e_(M-1)) in FP64 (it nearly cancels on fine grids).
        double b_sep = 1., bl_sep = 0., bu_sep = 0., bl_first = 0., bu_last = 0.;
        double L1 = 0., Llast = 0., R1 = 0., Rlast = 0.;
        {
            Walk wa = up(walk_at(j0 - 1), j0), wd = down(walk_at(j0 + M), j0 + M - 1);
            // the spacings behind each walk and their reciprocals
            double da = wa.dx, dd = wd.dx, ida = uniform ? iu_u : rcp(da), iud = uniform ? iu_u : rcp(dd);
            double idp = 1., bup = 0., fa = 0., pua = 1., suma = 0.;  // ascending: 1/d, bu, f, prod(-u), sum
            double iep = 1., blp = 0., fd = 0., pud = 1., sumd = 0.;  // descending
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
                    if (j < N) {
                        al = alpha_of(j, iu, im);
                        be = beta_of(j, im, ida);
                        bb = sub(add(1., add(al, be)), gamma);
                    }
                    store(i, x_of(wa), wa.c, al, be);
                    if (i == 0) {
                        bl_sep = -be;
                        b_sep = bb;
                        bu_sep = -al;
                    } else {
                        if (i == 1) bl_first = -be;
                        const double l = i == 1 ? 0. : -mul(be, idp);
                        const double d = fma(-l, bup, bb);
                        fa = i == 1 ? -be : -mul(l, fa);
                        if (i < P) {
                            const double r = rcp(d), u = -mul(al, r);
                            fit = fit && isfinite(r);
                            if (writer) {
                                tL(i) = (float)l;
                                tID(i) = (float)r;
                                tU(i) = (float)u;
                            }
                            suma = fma(mul(pua, fa), r, suma);
                            pua = -mul(pua, u);
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
                    if (j < N) {
                        al = alpha_of(j, iud, im);
                        be = beta_of(j, im, idn);
                        bb = sub(add(1., add(al, be)), gamma);
                    }
                    store(id_, x_of(wd), wd.c, al, be);
                    if (i == 1) bu_last = -al;
                    const double m = i == 1 ? 0. : -mul(al, iep);
                    const double r = rcp(fma(-m, blp, bb)), u = -mul(be, r);
                    fit = fit && isfinite(r);
                    fd = i == 1 ? -al : -mul(m, fd);
                    if (writer) {
                        tL(id_) = (float)m;
                        tID(id_) = (float)r;
                        tU(id_) = (float)u;
                    }
                    sumd = fma(mul(pud, fd), r, sumd);
                    pud = -mul(pud, u);
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
            fd = P > 1 ? -mul(mP, fd) : buP;
            if (writer) {
                tL(P) = (float)lP;
                tID(P) = (float)ig;
                tU(P) = (float)mP;
            }
            const double xl = mul(fa, ig), xr = mul(fd, ig);  // the spikes at the pivot
            L1 = fma(pua, xl, suma);
            Llast = mul(pud, xl);
            R1 = mul(pua, xr);
            Rlast = fma(pud, xr, sumd);
        }
        if (writer) {
            // spikes L = B_I^-1 (bl_1 e_1), R = B_I^-1 (bu_(M-1) e_(M-1)) by the steps' own solve
            auto spike = [&](float v1, float vn, int f) {
                float fa = 0.f, ga = 0.f;  // elimination results that reach the pivot
                float v[M];
#pragma unroll
                for (int i = 0; i < M; ++i) v[i] = 0.f;
                v[1] += v1;
                v[M - 1] += vn;
#pragma unroll
                for (int jj = 0; jj < P - 1; ++jj) {
                    const int it = 1 + jj, ib = M - 1 - jj;
                    fa = fmaf(-tL(it), fa, v[it]);
                    v[it] = fa;
                    ga = fmaf(-tL(ib), ga, v[ib]);
                    v[ib] = ga;
                }
                v[P] = fmaf(-tU(P), ga, fmaf(-tL(P), fa, v[P])) * tID(P);
#pragma unroll
                for (int jj = 0; jj < P - 1; ++jj) {
                    const int it = P - 1 - jj, ib = P + 1 + jj;
                    v[it] = fmaf(-tU(it), v[it + 1], v[it] * tID(it));
                    v[ib] = fmaf(-tU(ib), v[ib - 1], v[ib] * tID(ib));
                }
#pragma unroll
                for (int i = 1; i < M; ++i) (f ? tSR(i) : tSL(i)) = v[i];
            };
            spike((float)bl_first, 0.f, 0);
            spike(0.f, (float)bu_last, 1);
        }
        // separator system: warp-local cyclic reduction (multipliers in FP32), and for W > 1
        // the responses to the neighbours' values and the inverse of the boundary system
        float ka[5], kc[5], ib, rq = 0.f, rs = 0.f;
        float sl_m = 0.f, sr_m = 0.f;  // spikes of the previous lane's last node (warp boundaries)
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
                    sl_m = (float)Lprev;
                    sr_m = (float)Rprev;
                }
                if (k == 31) {
                    e[5 * warp + 2] = vq;
                    e[5 * warp + 3] = vs;
                    // the spikes as this lane's steps use them (the next warp repeats its update)
                    xs[2 * warp] = tSL(M - 1);
                    xs[2 * warp + 1] = tSR(M - 1);
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

        // ------------------------------------------------------------ time steps
        float2 H[P], L[P];
#pragma unroll
        for (int kk = 0; kk < P; ++kk) {
            const float4 p = PPt[kk * NL];
            H[kk] = f2(p.x, p.y);
            L[kk] = f2(p.z, p.w);
        }
        // no floor on the last node and on the padding
#pragma unroll
        for (int kk = 0; kk < P; ++kk) {
            const int na = j0 + (kk == 0 ? 0 : P - kk), nb = j0 + P + kk;
            if (na >= N - 1) PPt[kk * NL].x = -INFINITY;
            if (nb >= N - 1) PPt[kk * NL].y = -INFINITY;
        }
        const Split gs = split(gamma);
        const float2 gh = f2(gs.h, gs.h), gl = f2(gs.l, gs.l);
        // uniform grids of full lanes: the interior multipliers
        float2 cAh{}, cAl{}, cBh{}, cBl{};
        if constexpr (kUni) {
            const double al = alpha_of(1, iu_u, im_u), be = beta_of(1, im_u, iu_u);
            const Split sa = split(al), sb = split(be);
            cAh = f2(sa.h, sb.h);
            cAl = f2(sa.l, sb.l);
            cBh = f2(sb.h, sa.h);
            cBl = f2(sb.l, sa.l);
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
        // B x = y in FP32, in place on the slots; s1: x of the next lane's separator, um: x of
        // the previous lane's last node
        auto solve = [&](float2 (&y)[P], int which, float& s1, float& um) {
            phase_edge();
            float2 F = f2(0.f, 0.f);
#pragma unroll
            for (int kk = P - 1; kk >= 1; --kk) {
                F = fma2(neg(T1[kk * kStride]), F, y[kk]);
                y[kk] = F;
            }
            const float4 p2 = T2[0], p3 = T3[0];
            const float2 p1 = T1[0];
            const float yP = fmaf(-p2.w, F.y, fmaf(-p1.y, F.x, y[0].y)) * p2.y;
            float2 X = f2(yP, yP);
#pragma unroll
            for (int kk = 1; kk < P; ++kk) {
                const float4 q = T2[kk * kStride];
                X = fma2(neg(f2(q.z, q.w)), X, mul2(y[kk], f2(q.x, q.y)));
                y[kk] = X;
            }
            const float y_last = X.y, y_first = X.x;  // nodes M-1 and 1 (the pivot when P = 1)
            float ylp = __shfl_up_sync(kAll, y_last, 1);
            if (k == 0) ylp = 0.f;
            float rho = fmaf(-buf, y_first, fmaf(-blf, ylp, y[0].x));
#pragma unroll
            for (int lv = 0; lv < 5; ++lv) {
                const float rm = __shfl_up_sync(kAll, rho, 1 << lv), rp = __shfl_down_sync(kAll, rho, 1 << lv);
                rho = fmaf(-kc[lv], rp, fmaf(-ka[lv], rm, rho));
            }
            float s = rho * ib;
            if constexpr (W == 1) {
                s1 = __shfl_down_sync(kAll, s, 1);
                if (k == 31) s1 = 0.f;
                phase_edge();
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
                const float sl0 = __shfl_sync(kAll, sl_m, 0);
                const float Q = warp > 0 ? fmaf(-sl0, bl_, yl) : 0.f, Sr = warp < W - 1 ? ar : 0.f;
                s = fmaf(-rs, Sr, fmaf(rq, Q, s));
                if (k == 0 && warp > 0) s = a_;
                if (k == 31 && warp < W - 1) s = b_;
                s1 = __shfl_down_sync(kAll, s, 1);
                if (k == 31) s1 = Sr;
                // the previous warp's last node, by the operations its owner uses below
                um = fmaf(-a_, sr_m, fmaf(-bl_, sl_m, yl));
            }
            const float2 ms = f2(-s, -s), ms1 = f2(-s1, -s1);
#pragma unroll
            for (int kk = 1; kk < P; ++kk) {
                const float4 q = T3[kk * kStride];
                y[kk] = fma2(ms1, f2(q.z, q.w), fma2(ms, f2(q.x, q.y), y[kk]));
            }
            y[0] = f2(s, fmaf(-s1, p3.w, fmaf(-s, p3.y, yP)));
            const float u_last = P > 1 ? y[P - 1].y : y[0].y;
            const float up = __shfl_up_sync(kAll, u_last, 1);
            if (k > 0) um = up;
            if (K == 0) um = 0.f;
        };

        if (run) {
            for (int step = 1; step < TL; ++step) {
                // V of the neighbours: node -1 and node M
                const float2 last = P > 1 ? f2(H[P - 1].y, L[P - 1].y) : f2(H[0].y, L[0].y);
                float Hm = __shfl_up_sync(kAll, last.x, 1), Lm = __shfl_up_sync(kAll, last.y, 1);
                float Hp = __shfl_down_sync(kAll, H[0].x, 1), Lp = __shfl_down_sync(kAll, L[0].x, 1);
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
                        Hm = xe[4 * warp - 2];
                        Lm = xe[4 * warp - 1];
                    }
                    if (k == 31 && warp < W - 1) {
                        Hp = xe[4 * warp + 4];
                        Lp = xe[4 * warp + 5];
                    }
                }
                if (K == 0) Hm = Lm = 0.f;
                if (K == NL - 1) Hp = Lp = 0.f;
                phase_edge();

                // 1. u0 = B^-1 A' V in FP32.  D_k = V of slot k-1 minus V of slot k (the pivot
                // in both components before slot 1, nodes 0 and M after slot P-1)
                float2 y[P];
                float s1, um = 0.f;
                {
                    float2 Dc = f2(0.f, 0.f), D1 = f2(0.f, 0.f);
#pragma unroll
                    for (int kk = 1; kk <= P; ++kk) {
                        const float2 hu = kk == 1 ? f2(H[0].y, H[0].y) : H[kk - 1];
                        const float2 lu = kk == 1 ? f2(L[0].y, L[0].y) : L[kk - 1];
                        const float2 hd = kk == P ? f2(H[0].x, Hp) : H[kk];
                        const float2 ld = kk == P ? f2(L[0].x, Lp) : L[kk];
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
                    const float E = (H[0].x - Hm) + (L[0].x - Lm);
                    y[0] = fma2(A, f2(Dc.x, D1.y), fma2(neg(B), f2(E, D1.x), mul2(gh, H[0])));
                }
                solve(y, 0, s1, um);

                // 2., 3. W = V + u0 and r = A' W - u0
                float2 u0[P];
                phase_edge();
                {
                    const PP2 w0 = shifted(H[0], L[0], y[0]);
                    const PP2 wn = shifted(f2(Hm, Hp), f2(Lm, Lp), f2(um, s1));  // nodes -1 and M
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
                        const PP2 Dn = pair_diff(wc, wk);
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
                    const PP2 E = pair_diff(w0, {f2(wn.h.x, 0.f), f2(wn.l.x, 0.f)});
                    float2 Ah, Al, Bh, Bl;
                    coef_h(0, Ah, Bh);
                    coef_l(0, Al, Bl);
                    const PP2 X = {f2(Dc.h.x, D1.h.y), f2(Dc.l.x, D1.l.y)}, Z = {f2(E.h.x, D1.h.x), f2(E.l.x, D1.l.x)};
                    y[0] = pair_residual(Ah, Al, X, Bh, Bl, Z, gh, gl, w0, u0[0]);
                }
                // 4. e = B^-1 r, V' = max(V + 2 u0 + 2 e, p)
                solve(y, 1, s1, um);
                phase_edge();
#pragma unroll
                for (int kk = 0; kk < P; ++kk) {
                    float2 s, e;
                    two_sum(H[kk], add2(u0[kk], u0[kk]), s, e);
                    const float2 l = fma2(f2(2.f, 2.f), y[kk], add2(L[kk], e));
                    H[kk] = add2(s, l);
                    L[kk] = sub2(l, sub2(H[kk], s));
                    if (amer) {
                        const float4 p = PPt[kk * NL];
                        const float2 d = add2(sub2(H[kk], f2(p.x, p.y)), sub2(L[kk], f2(p.z, p.w)));
                        if (d.x < 0.f) {
                            H[kk].x = p.x;
                            L[kk].x = p.z;
                        }
                        if (d.y < 0.f) {
                            H[kk].y = p.y;
                            L[kk].y = p.w;
                        }
                    }
                }
            }
        }
        // ------------------------------------------------------------ result
        bool fin = run;
#pragma unroll
        for (int kk = 0; kk < P; ++kk) fin = fin && isfinite(H[kk].x) && isfinite(H[kk].y);
        fin = __all_sync(kAll, fin);
        if constexpr (W > 1) fin = __syncthreads_and(fin) != 0;
        if (fin) {
            double* V = vout + shape_row(sh, pde);
#pragma unroll
            for (int kk = 0; kk < P; ++kk) {
                const int na = j0 + (kk == 0 ? 0 : P - kk), nb = j0 + P + kk;
                if (na < N) V[na] = (double)H[kk].x + (double)L[kk].x;
                if (nb < N) V[nb] = (double)H[kk].y + (double)L[kk].y;
            }
        }
        if (K == 0) {
            pde_status[pde] = bad ? KWG_STATUS_BAD_INPUT : KWG_STATUS_OK;
            if (!fin && !bad) rescue[atomicAdd(&counters[2], 1)] = pde;
        }
    }
}

namespace {

template <int M, bool kUni, int W>
int& per_sm_pair64()
{
    static int v = 1;
    return v;
}

template <int M, bool kUni, int W>
void prepare_pair64_variant()
{
    constexpr size_t smem = Lay<M, kUni, W>::kBytes;
    cudaFuncSetAttribute(fd1d_solve_pair64<M, kUni, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fd1d_solve_pair64<M, kUni, W>, 32 * W, smem);
    per_sm_pair64<M, kUni, W>() = per_sm < 1 ? 1 : per_sm;
}

template <int M, bool kUni, int W>
void launch_pair64_variant(const PdeBatch& b, const Fd1dShape& sh, double* vout, int32_t* pde_status, int* counters,
                           int32_t* rescue, int sms, cudaStream_t stream)
{
    const int cap = sms * per_sm_pair64<M, kUni, W>();
    fd1d_solve_pair64<M, kUni, W><<<b.m < cap ? b.m : cap, 32 * W, Lay<M, kUni, W>::kBytes, stream>>>(
        b, sh, vout, pde_status, counters, rescue);
}

// Warps per PDE.  Enough PDEs to give every scheduler a warp: as few as the registers allow
// (more warps repeat the separator solve) -- one up to 1024 nodes, two on 1024-node grids
// whose tables are per node (45 KB per PDE: five PDEs per SM, so ten warps instead of five),
// four beyond.  Fewer PDEs: twice the warps while every warp still has a scheduler to
// itself, up to four (at eight, or below two nodes per lane, the exchange costs more than
// the shorter chains save).  Measured, ms (512 steps, density 0.25): 12 PDEs of 512 nodes with
// 1/2/4/8 warps 0.76/0.59/0.50/0.61, 300 of them 0.76/0.62/0.63/0.93, 600 of them
// 0.82/0.88/1.01; 8192 PDEs of 1024 nodes 18.4/15.0/17.1/28.2, on the uniform grid (1024
// steps) 24.2/25.1/29.4/51.0.
int pair64_warps(int m1, bool uni, int m, int sms)
{
    int w = m1 == 64 ? 4 : m1 == 32 && !uni ? 2 : 1;
    while (m1 >= 8 && w < 4 && (long long)m * 2 * w <= 4ll * sms) w *= 2;
    return w;
}

// (nodes per lane, warps per PDE) for grids of any kind, and the one for full uniform grids only
#define KWG_PAIR64_SHAPES(X) \
    X(2, 1) X(4, 1) X(8, 1) X(16, 1) X(4, 2) X(8, 2) X(16, 2) X(2, 4) X(4, 4) X(8, 4) X(16, 4)

}  // namespace

void fd1d_pair64_prepare(int)
{
#define X(MM, WW)                           \
    prepare_pair64_variant<MM, false, WW>(); \
    prepare_pair64_variant<MM, true, WW>();
    KWG_PAIR64_SHAPES(X)
#undef X
    prepare_pair64_variant<32, true, 1>();
}

size_t fd1d_pair64_work_bytes(int m, long long nodes) { return (size_t)nodes * sizeof(double) + (size_t)m * 4; }

int fd1d_pair64_launch(const PdeBatch& b, const AssetBatch& a, const Fd1dShape& sh, double* vout, int32_t* rescue,
                       int32_t* pde_status, int* counters, double* prices, int32_t* status, int device,
                       cudaStream_t stream, const SolveEvents* ev)
{
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int m1 = fd1d_fp32_nodes_per_lane(sh.x_dim);
    if (m1 < 0) return -1;
    const bool uni = sh.uniform && (sh.pde_x ? sh.full_lanes : sh.x_dim == 32 * m1);
    const int W = pair64_warps(m1, uni, b.m, sms), M = m1 / W;
    cudaMemsetAsync(counters, 0, 4 * sizeof(int), stream);
    if (ev) cudaEventRecord(ev->start, stream);
    if (M == 32) launch_pair64_variant<32, true, 1>(b, sh, vout, pde_status, counters, rescue, sms, stream);
#define X(MM, WW)                                                                                        \
    if (M == MM && W == WW) {                                                                            \
        if (uni)                                                                                         \
            launch_pair64_variant<MM, true, WW>(b, sh, vout, pde_status, counters, rescue, sms, stream); \
        else                                                                                             \
            launch_pair64_variant<MM, false, WW>(b, sh, vout, pde_status, counters, rescue, sms, stream); \
    }
    KWG_PAIR64_SHAPES(X)
#undef X
    int launches = 1 + fd1d_pcr64_rescue(b, sh, vout, rescue, pde_status, counters, sms, stream);
    if (ev) cudaEventRecord(ev->stop, stream);
    if (a.n > 0) {
        fd1d_interp_rows<<<(a.n + 127) / 128, 128, 0, stream>>>(b, a, sh, vout, pde_status, prices, status);
        ++launches;
    }
    return launches;
}

}  // namespace kwg
