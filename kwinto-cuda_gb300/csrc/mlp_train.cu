// mlp_train.cu -- loss and gradients of one minibatch in one tcgen05 kernel: forward,
// backward and weight gradients of a 64-row tile without leaving the SM.
//
// The layer-by-layer pass it replaces was bound by latency and by its own traffic: 27
// launches per minibatch, each with 32 or 16 CTAs of 128 threads that staged their operands
// through registers and wrote activations, SiLU', their transposes and dZ to global memory, one
// row per thread.  A 4096-row minibatch took 0.79 ms a call; this kernel's 64 CTAs keep
// everything on chip and only add 82 thousand gradient sums each to global memory: 0.065 ms
// a call.  It is bound by the latency of its eight dependent MMA-and-epilogue stages.
//
// Channels in lanes.  Every product is formed with the channels along the MMA's M (the TMEM
// lanes) and the rows along N, so a thread owns one channel of 32 rows: biases, the head's weight,
// the bias gradients and dW5 are scalars of the thread.  All operands are shared-memory tiles
// that are written once and read in either direction (the descriptors' K-major and MN-major
// forms): W serves z = W a and dA = W^T dZ, an activation tile serves the next layer and dW,
// dZ serves dA and dW.
//   z_l [out][row]  = W_l (a_hi + a_lo)       K-major W, K-major a
//   dA  [in][row]   = W_l^T dZ_l              MN-major W, K-major dZ
//   dW_l [out][in]  = sum_row dZ_l a_hi       MN-major dZ, MN-major a
// TMEM holds the four z (64 columns each; SiLU' is taken from them on the way back), dA (64) and
// two dW accumulators of 128 columns, the second over z_3 and z_4 once they are consumed, so the
// sums of one layer go out while the next layer's MMAs run.
//
// Roundings are those of the layer-by-layer pass: activations enter as BF16 pairs (weight
// gradients take the high part), W, dY and dZ as BF16, accumulation and everything else FP32.
// Every MMA completion wait is bounded (mlp_fused.cu).
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mlp.h"
#include "mlp_math.cuh"
#include "tc.cuh"
#include "tma.cuh"

namespace kwg {

namespace {

constexpr int kRows = 64, kThreads = 256, kW = kMlpWidth;
constexpr int kK1 = 16;  // layer-1 K: features hi 0..4, lo 5..9, zeros
constexpr uint32_t kW1Bytes = kW * kK1 * 2, kWBytes = kW * kW * 2, kXBytes = kRows * kK1 * 2;
// Activation and dZ tiles: core matrices (8 rows x 16 bytes) 160 bytes apart along the channels, so
// that the 32 channels of a warp's store fall into different banks.
constexpr uint32_t kCore = 160, kRow8 = (kW / 8) * kCore, kABytes = (kRows / 8) * kRow8;
constexpr uint32_t kOffW1 = 0, kOffW = kOffW1 + kW1Bytes, kOffX = kOffW + 3 * kWBytes, kOffA = kOffX + kXBytes,
                   kOffZ = kOffA + 3 * kABytes,  // a_lo on the way forward, dZ on the way back
                   kOffBias = kOffZ + kABytes, kOffHead = kOffBias + 4 * kW * 4, kOffY = kOffHead + kW * 4,
                   kOffG = kOffY + 4 * kRows * 4, kOffMisc = kOffG + kRows * 4, kSmem = kOffMisc + 64;
// TMEM columns
constexpr uint32_t kColZ = 0, kColA = 256, kColW0 = 320, kColW1 = 128, kColWIn = 448, kTmem = 512;

__device__ __forceinline__ uint32_t act_offset(int row, int ch)
{
    return (uint32_t)(row >> 3) * kRow8 + (uint32_t)(ch >> 3) * kCore + (uint32_t)((row & 7) * 16 + (ch & 7) * 2);
}

// Sums over the 32 lanes of 32 values: lane i returns the sum of v[i] (31 shuffles).
__device__ __forceinline__ float lane_sums(float (&v)[32], int lane)
{
#pragma unroll
    for (int off = 16; off >= 1; off /= 2) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < off; ++i) {
            const float send = up ? v[i] : v[i + off], keep = up ? v[i + off] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    return v[0];
}

// Rows of the accumulator at TMEM column `col` (64 columns per thread) into the gradient matrix.
__device__ __forceinline__ void add_rows(float* __restrict__ dst, uint32_t taddr)
{
#pragma unroll
    for (int c = 0; c < 64; c += 32) {
        float v[32];
        tc::tmem_ld32(taddr + (uint32_t)c, v);
#pragma unroll
        for (int i = 0; i < 32; i += 4)
            atomicAdd(reinterpret_cast<float4*>(dst + c + i), make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
    }
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 1)
    mlp_grad_fused(const float* __restrict__ x, const float* __restrict__ t, const float* __restrict__ fl,
                   const int32_t* __restrict__ idx, int b, const __nv_bfloat16* __restrict__ wb,
                   const float* __restrict__ params, float* __restrict__ g, double* __restrict__ loss,
                   int* __restrict__ error)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int ch = (warp & 3) * 32 + lane, half = warp >> 2;  // this thread's channel, and its rows half*32 ..
    uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + kOffMisc);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + kOffMisc + 8);
    float* ysum = reinterpret_cast<float*>(sm + kOffY);
    float* grow = reinterpret_cast<float*>(sm + kOffG);

    // resident weights, as mlp_fused.cu
    auto store_core = [&](uint32_t base, int kc, int row, int k, uint4 v) {
        *reinterpret_cast<uint4*>(sm + base + tc::core_offset(row, k, kc)) = v;
    };
    for (int v = tid; v < kW * (kK1 / 8); v += kThreads)
        store_core(kOffW1, kK1, v / 2, (v % 2) * 8,
                   *reinterpret_cast<const uint4*>(wb + (size_t)(v / 2) * kMlpInK + (v % 2) * 8));
#pragma unroll
    for (int l = 0; l < 3; ++l) {
        const __nv_bfloat16* src = wb + (size_t)(l + 1) * kMlpFwdSlot;
#pragma unroll
        for (int i = 0; i < kW * (kW / 8) / kThreads; ++i) {
            const int v = tid + i * kThreads, row = v / (kW / 8), kq = v % (kW / 8);
            store_core(kOffW + l * kWBytes, kW, row, kq * 8,
                       *reinterpret_cast<const uint4*>(src + (size_t)row * kMlpHidK + kq * 8));
        }
    }
    float bias[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) bias[l] = params[kMlpWeights + l * kW + ch];
    const float head = __bfloat162float(wb[4 * kMlpFwdSlot + ch]), head_b = params[kMlpWeights + 4 * kW];
    if (warp == 0) {
        tc::tmem_alloc(smem_addr(tslot), kTmem);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(mbar, 1);
        fence_mbar_init();
    }
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot, tl = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t s0 = smem_addr(sm);
    const uint32_t i_fwd = tc::idesc_bf16_f32(kW, kRows), i_dx = i_fwd | tc::kMajorMnA,
                   i_dw = tc::idesc_bf16_f32(kW, kW) | tc::kMajorMnA | tc::kMajorMnB,
                   i_dw1 = tc::idesc_bf16_f32(kW, kK1) | tc::kMajorMnA | tc::kMajorMnB;
    uint32_t phase = 0;
    bool ok = true, pending = false;
    auto wait = [&]() -> bool {
        ok = mbar_wait(mbar, phase) && ok;
        phase ^= 1u;
        ok = __syncthreads_and(ok);
        if (ok) pending = false;
        tc::fence_after_sync();
        return ok;
    };
    // before an MMA: this thread's shared-memory writes and TMEM reads come first
    auto ready = [&]() {
        tc::fence_proxy_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        pending = true;
    };
    // dA = W_(l+1)^T dZ (l = 1..3: the activations a_l) and dW_(l+1) += dZ a_l^T into column `col`
    auto back_mma = [&](int l, uint32_t col) {
        tc::fence_after_sync();
        const uint32_t w = s0 + kOffW + (uint32_t)(l - 1) * kWBytes, z = s0 + kOffZ, al = s0 + kOffA + (uint32_t)(l - 1) * kABytes;
#pragma unroll
        for (int kk = 0; kk < kW / 16; ++kk)
            tc::mma_bf16(tmem + kColA, tc::smem_desc(w + kk * 2 * (kW / 8) * 128, (kW / 8) * 128, 128),
                         tc::smem_desc(z + kk * 2 * kCore, kCore, kRow8), i_dx, kk > 0);
#pragma unroll
        for (int kk = 0; kk < kRows / 16; ++kk)
            tc::mma_bf16(tmem + col, tc::smem_desc(z + kk * 2 * kRow8, kRow8, kCore),
                         tc::smem_desc(al + kk * 2 * kRow8, kRow8, kCore), i_dw, kk > 0);
        tc::commit(smem_addr(mbar));
    };

    for (int tile = blockIdx.x; tile * kRows < b; tile += gridDim.x) {
        const int r0 = tile * kRows;
        float tgt = 0.f, flo = -kNoFloor;
        if (tid < kRows) {
            const int r = r0 + tid;
            float f[kMlpIn] = {0.f, 0.f, 0.f, 0.f, 0.f};
            if (r < b) {
                const int src = idx ? idx[r] : r;
#pragma unroll
                for (int c = 0; c < kMlpIn; ++c) f[c] = x[(size_t)src * kMlpIn + c];
                tgt = t[src];
                if (fl) flo = fl[src];
            }
            __align__(16) __nv_bfloat16 xr[kK1];
            split_features<kK1>(f, xr);
            store_core(kOffX, kK1, tid, 0, *reinterpret_cast<const uint4*>(xr));
            store_core(kOffX, kK1, tid, 8, *reinterpret_cast<const uint4*>(xr + 8));
        }
        ready();
        if (tid == 0) {
            tc::fence_after_sync();
            tc::mma_bf16(tmem + kColZ, tc::smem_desc(s0 + kOffW1, 128, (kK1 / 8) * 128),
                         tc::smem_desc(s0 + kOffX, 128, (kK1 / 8) * 128), i_fwd, false);
            tc::commit(smem_addr(mbar));
        }
        // ---- forward: layers 1..3, their activations as hi and lo tiles
        float z[32];
#pragma unroll 1
        for (int l = 0; l < 4; ++l) {
            if (!wait()) break;
            tc::tmem_ld32(tl + kColZ + (uint32_t)(l * kRows + half * 32), z);
            const float bl = l == 0 ? bias[0] : l == 1 ? bias[1] : l == 2 ? bias[2] : bias[3];
#pragma unroll
            for (int j = 0; j < 32; ++j) z[j] += bl;
            if (l == 3) break;
            unsigned char* hi_t = sm + kOffA + l * kABytes;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float a = silu_f(z[j]);
                const __nv_bfloat16 hi = __float2bfloat16(a);
                const uint32_t o = act_offset(half * 32 + j, ch);
                *reinterpret_cast<__nv_bfloat16*>(hi_t + o) = hi;
                *reinterpret_cast<__nv_bfloat16*>(sm + kOffZ + o) = __float2bfloat16(a - __bfloat162float(hi));
            }
            ready();
            if (tid == 0) {
                tc::fence_after_sync();
                const uint32_t w = s0 + kOffW + (uint32_t)l * kWBytes;
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    const uint32_t a = part == 0 ? s0 + kOffA + (uint32_t)l * kABytes : s0 + kOffZ;
#pragma unroll
                    for (int kk = 0; kk < kW / 16; ++kk)
                        tc::mma_bf16(tmem + kColZ + (uint32_t)((l + 1) * kRows),
                                     tc::smem_desc(w + kk * 256, 128, (kW / 8) * 128),
                                     tc::smem_desc(a + kk * 2 * kCore, kCore, kRow8), i_fwd, part > 0 || kk > 0);
                }
                tc::commit(smem_addr(mbar));
            }
        }
        if (!ok) break;
        // ---- the head, the loss and dY
        {
            float v[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = head * silu_f(z[j]);
            ysum[(warp & 3) * kRows + half * 32 + lane] = lane_sums(v, lane);
        }
        __syncthreads();
        if (tid < kRows) {
            const float y = (ysum[tid] + ysum[kRows + tid]) + (ysum[2 * kRows + tid] + ysum[3 * kRows + tid]) + head_b;
            float dy = 0.f;
            double l2 = 0.;
            if (r0 + tid < b) {
                const float e = flo > -kNoFloor ? fmaxf(0.f, y - flo) : y - tgt;
                dy = 2.f * e / (float)b;
                l2 = (double)e * (double)e / (double)b;
            }
            grow[tid] = __bfloat162float(__float2bfloat16(dy));
            for (int off = 16; off >= 1; off /= 2) {
                dy += __shfl_xor_sync(0xffffffffu, dy, off);
                l2 += __shfl_xor_sync(0xffffffffu, l2, off);
            }
            if (lane == 0) {
                atomicAdd(loss, l2);
                atomicAdd(g + kMlpWeights + 4 * kW, dy);
            }
        }
        __syncthreads();
        // ---- layer 4: dA = dY W5, dW5, dZ4
        {
            float dw5 = 0.f, db = 0.f;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float gr = grow[half * 32 + j];
                dw5 = fmaf(gr, __bfloat162float(__float2bfloat16(silu_f(z[j]))), dw5);
                const float dz = gr * head * dsilu_f(z[j]);
                db += dz;
                *reinterpret_cast<__nv_bfloat16*>(sm + kOffZ + act_offset(half * 32 + j, ch)) = __float2bfloat16(dz);
            }
            atomicAdd(g + (size_t)4 * kW * kW + ch, dw5);
            atomicAdd(g + kMlpWeights + 3 * kW + ch, db);
        }
        ready();
        if (tid == 0) back_mma(3, kColW0);
        // ---- layers 3..1
#pragma unroll 1
        for (int l = 3; l >= 1; --l) {
            if (!wait()) break;
            float da[32];
            tc::tmem_ld32(tl + kColZ + (uint32_t)((l - 1) * kRows + half * 32), z);
            tc::tmem_ld32(tl + kColA + (uint32_t)(half * 32), da);
            const float bl = l == 3 ? bias[2] : l == 2 ? bias[1] : bias[0];
            float db = 0.f;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float dz = da[j] * dsilu_f(z[j] + bl);
                db += dz;
                *reinterpret_cast<__nv_bfloat16*>(sm + kOffZ + act_offset(half * 32 + j, ch)) = __float2bfloat16(dz);
            }
            ready();
            if (tid == 0) {
                if (l > 1) {
                    back_mma(l - 1, l == 3 ? kColW1 : kColW0);
                } else {
                    tc::fence_after_sync();
#pragma unroll
                    for (int kk = 0; kk < kRows / 16; ++kk)
                        tc::mma_bf16(tmem + kColWIn, tc::smem_desc(s0 + kOffZ + kk * 2 * kRow8, kRow8, kCore),
                                     tc::smem_desc(s0 + kOffX + kk * 2 * (kK1 / 8) * 128, (kK1 / 8) * 128, 128), i_dw1,
                                     kk > 0);
                    tc::commit(smem_addr(mbar));
                }
            }
            // dW_(l+1) while those MMAs run
            atomicAdd(g + kMlpWeights + (l - 1) * kW + ch, db);
            add_rows(g + (size_t)l * kW * kW + (size_t)ch * kW + half * 64,
                     tl + (l == 2 ? kColW1 : kColW0) + (uint32_t)(half * 64));
        }
        if (!ok || !wait()) break;
        if (half == 0) {
            float v[32];
            tc::tmem_ld32(tl + kColWIn, v);
#pragma unroll
            for (int c = 0; c < kMlpIn; ++c) atomicAdd(g + (size_t)ch * kW + c, v[c]);
        }
        tc::fence_before_sync();  // TMEM reads of this tile precede the next tile's MMAs
    }
    if (!ok) {
        if (tid == 0 && error) atomicExch(error, 1);
        if (pending) mbar_wait(mbar, phase ^ 1u);  // let the MMAs in flight finish before TMEM is freed
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, kTmem);
}

cudaError_t mlp_grad_set_smem_limit()
{
    return cudaFuncSetAttribute(mlp_grad_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
}

cudaError_t mlp_launch_grad(const float* x, const float* t, const float* fl, const int32_t* idx, int b,
                            const __nv_bfloat16* wb, const float* params, float* g, double* loss, int* error, int sms,
                            cudaStream_t st)
{
    if (const cudaError_t e = mlp_prepare_device(); e != cudaSuccess) return e;
    const int tiles = (b + kRows - 1) / kRows;
    mlp_grad_fused<<<tiles < sms ? tiles : sms, kThreads, kSmem, st>>>(x, t, fl, idx, b, wb, params, g, loss, error);
    return cudaGetLastError();
}

}  // namespace kwg
