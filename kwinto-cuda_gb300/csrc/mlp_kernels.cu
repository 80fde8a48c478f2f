// mlp_kernels.cu -- elementwise kernels of the MLP surrogate (the GEMM is in mlp_gemm.cu, the
// minibatch gradients in mlp_train.cu).  Layer inputs are BF16 (hi, lo) pairs and the forward
// weights are stored twice along K (layout in mlp.h).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kwg.h"
#include "mlp.h"
#include "mlp_math.cuh"

namespace kwg {

// Features, in-box flag and the analytic base price: Barone-Adesi-Whaley for
// American options, Black-Scholes for European ones.
__global__ void mlp_featurize(const kwg_option* __restrict__ opts, int n, MlpBox box, float* __restrict__ x,
                              uint8_t* __restrict__ inside, double* __restrict__ base)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const kwg_option o = opts[i];
    float f[kMlpIn];
    bool in = false;
    const OptionTerms terms = option_terms(o);
    features(o, terms, box, f, in);
    if (x)
#pragma unroll
        for (int c = 0; c < kMlpIn; ++c) x[(size_t)i * kMlpIn + c] = f[c];
    if (base) base[i] = base_price(o, terms);
    if (inside) inside[i] = in ? 1 : 0;
}

// One thread per row r < b_pad: split BF16 row of 64 (hi 0..4, lo 5..9, zeros).
__global__ void mlp_pack(const float* __restrict__ f, int b, int b_pad, __nv_bfloat16* __restrict__ x)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= b_pad) return;
    float fr[kMlpIn];
#pragma unroll
    for (int c = 0; c < kMlpIn; ++c) fr[c] = r < b ? f[(size_t)r * kMlpIn + c] : 0.f;
    __align__(16) __nv_bfloat16 row[kMlpInK];
    split_features<kMlpInK>(fr, row);
    uint4* dst = reinterpret_cast<uint4*>(x + (size_t)r * kMlpInK);
    const uint4* srcv = reinterpret_cast<const uint4*>(row);
#pragma unroll
    for (int q = 0; q < kMlpInK / 8; ++q) dst[q] = srcv[q];
}

// Adam on FP32 master parameters; the gradients are cleared for the next minibatch's sums.
__global__ void mlp_adam(float* __restrict__ p, float* __restrict__ g, float* __restrict__ m,
                         float* __restrict__ v, int n, float lr, float b1, float b2, float eps, float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    g[i] = 0.f;
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// BF16 copies of the weights: the K-doubled forward operands [W | W] (layer 1:
// inputs 0..4 at columns 0..4 and 5..9 of a 64-wide row) and the head row.  Grid (128
// rows, 5 layers), 128 threads.
__global__ void mlp_refresh(const float* __restrict__ w, __nv_bfloat16* __restrict__ wb)
{
    const int l = blockIdx.y;
    const int o = blockIdx.x, i = threadIdx.x;
    const size_t base = (size_t)l * kMlpWidth * kMlpWidth;
    const __nv_bfloat16 h = __float2bfloat16(w[base + (size_t)o * kMlpWidth + i]);
    __nv_bfloat16* slot = wb + (size_t)l * kMlpFwdSlot;
    if (l == 0) {
        if (i < kMlpInK) {
            const int src = i < kMlpIn ? i : i < 2 * kMlpIn ? i - kMlpIn : -1;
            slot[(size_t)o * kMlpInK + i] =
                src >= 0 ? __float2bfloat16(w[base + (size_t)o * kMlpWidth + src]) : __float2bfloat16(0.f);
        }
    } else if (l < 4) {
        slot[(size_t)o * kMlpHidK + i] = h;
        slot[(size_t)o * kMlpHidK + kMlpWidth + i] = h;
    } else if (o == 0) {
        slot[i] = h;  // head row: W5[0][i]
    }
}

void mlp_launch_featurize(const kwg_option* opts, int n, const MlpBox& box, float* x, uint8_t* inside, double* base,
                          cudaStream_t st)
{
    mlp_featurize<<<(n + 127) / 128, 128, 0, st>>>(opts, n, box, x, inside, base);
}

void mlp_launch_pack(const float* f, int b, int b_pad, __nv_bfloat16* x, cudaStream_t st)
{
    mlp_pack<<<(b_pad + 127) / 128, 128, 0, st>>>(f, b, b_pad, x);
}

void mlp_launch_adam(float* p, float* g, float* m, float* v, int n, float lr, float b1, float b2, float eps,
                     float c1, float c2, cudaStream_t st)
{
    mlp_adam<<<(n + 255) / 256, 256, 0, st>>>(p, g, m, v, n, lr, b1, b2, eps, c1, c2);
}

void mlp_launch_refresh(const float* w, __nv_bfloat16* wb, cudaStream_t st)
{
    mlp_refresh<<<dim3(kMlpWidth, kMlpLayers), kMlpWidth, 0, st>>>(w, wb);
}

}  // namespace kwg
