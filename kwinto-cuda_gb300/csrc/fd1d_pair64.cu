// fd1d_pair64.cu -- the FP64 theta-scheme solve (theta = 1/2) on the FP32 units: one to
// four warps per PDE, the whole PDE on chip, values as pairs of floats and one step of
// iterative refinement per time step.
//
// Why.  A warp-wide FP64 instruction holds its scheduler's FP64 unit for 64 cycles, a
// warp-wide FP32 one for 1.  The streaming kernel's three FP64 multiply-adds per node-step
// (fd1d_fp64.cu) therefore cost 6 scheduler cycles per node; the ~79 FP32 operations here
// cost 2.5, and their latency is 4 cycles instead of 64.
//
// Bound by the FP32 pipe (75 % busy at 1024 uniform nodes) and, for few PDEs, by the
// latency of the two separator solves per step.  Measured against the FP64 solvers that took
// these shapes before (whole calls): 32768 PDEs, 1024 x 1024 uniform, 192 -> 87 ms; 8192 PDEs,
// 1024 x 1024, density 0.25, 186 -> 27 ms; 777 PDEs, 1000 x 731, 12.4 -> 2.5 ms; 600 PDEs,
// 512 x 512, 2.50 -> 0.78 ms; 12 PDEs 2.35 -> 0.45 ms; 131072 uneven PDEs 340 -> 133 ms.
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
// difference form has no such drift.  Against stepping in 64-bit increments (48 to 2048 nodes, 40 to 2048 time levels,
// uniform and density 0.25, 64 to 32768 options): 3e-15 to 8e-13 where the FP64 solvers have 3e-15 to 6e-12, and
// nowhere more than they (1.05 times at 3.5e-15 at most).
//
// What it does not take: theta != 1/2, more than 2048 nodes, and -- PDE by PDE, found in
// the setup or at the end -- values beyond FP32's range, and grids that a drift crosses
// (|r - q - z^2/2| T above kMaxDrift half-widths), where the one-sided boundary rows of the
// scheme amplify whatever stands at the boundary by orders of magnitude.  Those PDEs go
// to a list that the FP64 kernel of fd1d_pcr64.cu works off in a launch of its own; a batch with many of
// them is not given to this solver (fp64_route.h).
#include "fd1d_onchip.cuh"

namespace kwg {

namespace {

// Warps per PDE.  Enough PDEs to give every scheduler a warp: as few as the registers allow
// (more warps repeat the separator solve) -- one up to 1024 nodes, two on 1024-node grids
// whose tables are per node (37 KB per PDE: six PDEs per SM, so twelve warps instead of six),
// four beyond.  Fewer PDEs: twice the warps while every warp still has a scheduler to
// itself, from 1024 nodes while they fit 12 to an SM, up to four (at eight, or below two nodes
// per lane, the exchange costs more than the shorter chains save).  Measured, ms with 1/2/4
// warps (256 steps): density 0.25, 150 PDEs of 512 nodes 0.359/0.277/0.226, 300 of them
// 0.361/0.281/0.295, 450 of them 0.361/0.392/0.383; uniform, 300 of 1024 nodes 0.645/0.418/0.393, 450 of
// them 0.655/0.578/0.524, 600 of them 0.672/0.596/0.684, 900 of them 0.967/0.809/1.000, 1200 of them
// 1.008/1.030/1.270; 8192 of 1024 nodes, density 0.25 (511 steps) -/13.7/16.1.
int pair64_warps(int m1, bool uni, int m, int sms)
{
    int w = m1 == 64 ? 4 : m1 == 32 && !uni ? 2 : 1;
    while (m1 >= 8 && w < 4 && (long long)m * 2 * w <= (m1 >= 32 ? 12ll : 4ll) * sms) w *= 2;
    return w;
}

// (nodes per lane, warps per PDE) for grids of any kind, and the one for full uniform grids only
#define KWG_PAIR64_SHAPES(X) \
    X(2, 1) X(4, 1) X(8, 1) X(16, 1) X(4, 2) X(8, 2) X(16, 2) X(2, 4) X(4, 4) X(8, 4) X(16, 4)

}  // namespace

void fd1d_pair64_prepare(int)
{
#define X(MM, WW)                           \
    prepare_onchip<MM, false, WW, true>(); \
    prepare_onchip<MM, true, WW, true>();
    KWG_PAIR64_SHAPES(X)
#undef X
    prepare_onchip<32, true, 1, true>();
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
    if (M == 32) launch_onchip<32, true, 1, true>(b, sh, vout, pde_status, counters, rescue, sms, stream);
#define X(MM, WW)                                                                                        \
    if (M == MM && W == WW) {                                                                            \
        if (uni)                                                                                         \
            launch_onchip<MM, true, WW, true>(b, sh, vout, pde_status, counters, rescue, sms, stream); \
        else                                                                                             \
            launch_onchip<MM, false, WW, true>(b, sh, vout, pde_status, counters, rescue, sms, stream); \
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
