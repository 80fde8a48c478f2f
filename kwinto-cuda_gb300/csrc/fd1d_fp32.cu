// fd1d_fp32.cu -- FP32 stepping with FP64-accurate state: the on-chip kernel (fd1d_onchip.cuh)
// with one FP32 solve per step, and the interpolation over rows of final values.
//
// Numerics.  The reference step B V' = E V (src/Math/kwFd1d.cpp:61-132) is taken in
// delta form,  V' = max(V + d, p)  with  B d = dt A V  (E = B + dt A), so FP32 only
// ever carries the small increment d, and over X = V - p, p the payoff:
//     B d = dt A X + q,   X' = max(X + d, 0),   q = dt A p.
// X is a float-float pair (hi + lo, ~48 significant bits).  The residual dt A X is formed from
// differences of the pairs, which are exact in FP32, with the operator written as
//     dt A X_j = c1 S_j + c2 (X_{j+1}-X_j) + c3 (X_j-X_{j-1}) + c4 X_j,
//     S_j = (X_{j+1}-X_j) - (X_j-X_{j-1}),
// c1 = dt axx l2, c2 = dt (axx (u2-l2) + ax im), c3 = dt ax im, c4 = dt a0 (the
// reference's inverse spacings, src/Math/kwFd1d.cpp:87-92), so rounding the
// coefficients to FP32 perturbs the PDE's coefficients by ~1e-7 relatively instead
// of breaking the cancellation of the second difference.  q uses the same rounded
// coefficients (fd1d_onchip.cuh).  The grid, c1..c4, the factors and
// the payoff are computed in FP64 (src/Pricer/kwFd1d.cpp:110-139); the final
// interpolation reads V = p + hi + lo in FP64.
//
// Over V itself a step compares with the payoff: three more packed operations per two nodes
// (23 against 20) and 16 bytes of tables per slot instead of the 8 of q.  Per 8192 PDEs: 1024
// nodes (1024 steps) 9.63 -> 8.59 ms, density 0.25 (512 steps) 6.90 -> 6.08; 4096 of 2048 (512 steps)
// 5.26 -> 4.36; and 7.60, 5.96, 4.36 with the registers that it freed (budget()).
#include "fd1d_onchip.cuh"

namespace kwg {

// One thread per asset, like fd1d_interp_fp64 but over a [pde][x_dim] array of V.
__global__ void fd1d_interp_rows(const PdeBatch b, const AssetBatch a, Fd1dShape sh, const double* __restrict__ vrow,
                                 const int32_t* __restrict__ pde_status, double* __restrict__ prices,
                                 int32_t* __restrict__ status)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n || (sh.left_streams && many_left(sh))) return;
    const int slot = a.pde[i];
    const int N = shape_x(sh, slot);
    const double s = a.s[i], k = a.k[i];
    int32_t st = pde_status[slot];
    if (!(s > 0.) || !(k > 0.) || !isfinite(s) || !isfinite(k)) st = KWG_STATUS_BAD_INPUT;
    double price = __longlong_as_double(0x7ff8000000000000ll);
    if (st == KWG_STATUS_OK) {
        Grid g;
        g.init(b.z[slot], b.t[slot], sh.scale, sh.density, N, sh.uniform);
        const double xs = log(dvd(s, k));
        int lo = 0, hi = N;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (g.x(mid) < xs)
                lo = mid + 1;
            else
                hi = mid;
        }
        if (lo == 0 || lo == N) {
            st = KWG_STATUS_OUT_OF_GRID;
        } else {
            const double* V = vrow + shape_row(sh, slot);
            const double xl = g.x(lo - 1), xh = g.x(lo);
            const double v = dvd(add(mul(sub(xh, xs), V[lo - 1]), mul(sub(xs, xl), V[lo])), sub(xh, xl));
            price = mul(k, v);
        }
    }
    // a solve that left a non-finite value where the price is read is a solver failure
    // (the FP32 path's float-float state overflows beyond ~3.4e38 x K)
    if (st == KWG_STATUS_OK && !isfinite(price)) {
        st = KWG_STATUS_SOLVER;
        price = __longlong_as_double(0x7ff8000000000000ll);
    }
    prices[i] = price;
    if (status) status[i] = st;
}

namespace {

// Warps per PDE by the batch size: one up to 512 nodes and on 1024-node uniform grids, two on
// 1024-node grids with tables per node and on 2048-node uniform ones, four on 2048-node grids
// with tables per node; twice as many while every warp still has a scheduler to itself, and
// from 1024 nodes (512 with tables per node) while they fit 12 to an SM.  Measured, ms with
// 1/2/4 warps: 256 steps, uniform grids of 512 nodes, 150 PDEs 0.130/0.114/0.104, 300 of them
// 0.130/0.116/0.129, 600 of them 0.135/0.149/0.194; of 1024 nodes, 300 of them 0.237/0.170/0.163, 900 of them
// 0.344/0.311/0.395, 1200 of them 0.364/0.436/0.528; 512 nodes at density 0.25, 600 of them 0.206/0.192/0.296; 511
// steps, 8192 PDEs of 1024 nodes, density 0.25, 5.86/5.25/6.59, uniform 3.77/4.41/5.82; 4096 PDEs of 2048 nodes
// -/6.22/5.87, uniform -/4.17/5.37.
int fp32_warps(int m1, bool uni, int m, int sms)
{
    int w = m1 == 64 ? (uni ? 2 : 4) : m1 == 32 && !uni ? 2 : 1;
    for (; m1 >= 8 && w < 4; w *= 2) {
        const bool shared = m1 >= 32 || (m1 == 16 && !uni && w == 1);
        if ((long long)m * 2 * w > (shared ? 12ll : 4ll) * sms) break;
    }
    return w;
}

// (nodes per lane, warps per PDE)
#define KWG_FP32_SHAPES(X) \
    X(2, 1) X(4, 1) X(8, 1) X(16, 1) X(32, 1) X(4, 2) X(8, 2) X(16, 2) X(32, 2) X(2, 4) X(4, 4) X(8, 4) X(16, 4)

}  // namespace

void fd1d_fp32_prepare(int)
{
#define X(MM, WW)                               \
    prepare_onchip<MM, false, WW, false>(); \
    prepare_onchip<MM, true, WW, false>();
    KWG_FP32_SHAPES(X)
#undef X
}

int fd1d_fp32_nodes_per_lane(int x_dim)
{
    int m = 2;
    while (32 * m < x_dim) m *= 2;
    return m <= 64 ? m : -1;
}

int fd1d_fp32_warps(int x_dim, int option_warps)
{
    const int m1 = fd1d_fp32_nodes_per_lane(x_dim);
    if (m1 < 8) return 1;
    const int w = option_warps > 4 ? 4 : option_warps;
    return m1 == 64 && w < 2 ? 2 : w;
}

size_t fd1d_fp32_work_bytes(int m, int x_dim) { return (size_t)m * x_dim * sizeof(double); }

int fd1d_fp32_launch(const PdeBatch& b, const AssetBatch& a, const Fd1dShape& sh, double* vout, int32_t* pde_status,
                     int* counters, double* prices, int32_t* status, int device, cudaStream_t stream,
                     const SolveEvents* ev)
{
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    // W warps per PDE (sh.option_warps, or by the rule), each lane owning M = m1 / W nodes, m1
    // the nodes per lane of the one-warp layout
    const int m1 = fd1d_fp32_nodes_per_lane(sh.x_dim);
    if (m1 < 0) return -1;
    const bool uni = sh.uniform && (sh.pde_x ? sh.full_lanes : sh.x_dim == 32 * m1);
    const int W = fd1d_fp32_warps(sh.x_dim, sh.option_warps > 0 ? sh.option_warps : fp32_warps(m1, uni, b.m, sms));
    const int M = m1 / W;
    cudaMemsetAsync(counters, 0, 4 * sizeof(int), stream);
    if (ev) cudaEventRecord(ev->start, stream);
#define X(MM, WW)                                                                                             \
    if (M == MM && W == WW) {                                                                                 \
        if (uni)                                                                                              \
            launch_onchip<MM, true, WW, false>(b, sh, vout, pde_status, counters, nullptr, sms, stream);      \
        else                                                                                                  \
            launch_onchip<MM, false, WW, false>(b, sh, vout, pde_status, counters, nullptr, sms, stream);     \
    }
    KWG_FP32_SHAPES(X)
#undef X
    if (ev) cudaEventRecord(ev->stop, stream);
    int launches = 1;
    if (a.n > 0) {
        fd1d_interp_rows<<<(a.n + 127) / 128, 128, 0, stream>>>(b, a, sh, vout, pde_status, prices, status);
        ++launches;
    }
    return launches;
}

}  // namespace kwg
