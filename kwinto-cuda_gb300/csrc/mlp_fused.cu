// mlp_fused.cu -- surrogate pricing in one persistent tcgen05 kernel: option in,
// price out, activations never leave the SM.
//
// One CTA per SM (512 threads: four warpgroups) keeps the BF16 weights of all layers in shared
// memory (core-matrix layout, tc.cuh) for its whole life and walks 128-option tiles:
//   * warpgroups 2 and 3 take the CTA's even and odd tiles, an option per thread: its
//     features as the split BF16 row (hi 0..4, lo 5..9) of the 128 x 16 input tile, and its analytic
//     base price (FP64 Black-Scholes and FP32 Barone-Adesi-Whaley critical price), both into
//     one of two shared-memory slots.  A warp waits for nothing but its slot;
//   * warpgroups 0 and 1 run the network: thread t serves row t % 128, the first warpgroup
//     accumulator columns 0..63 of it, the second 64..127 (a warp reads the TMEM lanes of its
//     rank in the warpgroup).  The epilogue of layers 1-3 reads the accumulator (tcgen05.ld), adds
//     the bias, applies SiLU and writes the activation as a BF16 pair into the hi and lo 128 x
//     128 tiles; thread 0 then issues 8 MMAs over hi and 8 over lo with the same weight operand
//     (the GEMM path's K-doubled [W | W] sums the same terms).  The layers alternate between two
//     TMEM accumulators, so the next tile's layer 1 (K = 16) is issued right behind layer 4 of this
//     one.  The layer-4 epilogue folds the 128 -> 1 head into an FP32 dot product in column order
//     (the first warpgroup sums columns 0..63, the second continues from its partial over 64..127,
//     as the GEMM path's epilogue does) and writes max(intrinsic, base + K y / y_scale).
// The arithmetic matches the layer-by-layer path (mlp_gemm.cu) step for step.
//
// With features, base price and layers in turn, a tile took the sum of three latency-bound chains:
// 3.09 ms for 10^6 options, issue slots 23 % busy.  Side by side: 1.37 ms, bound by the epilogues
// (SiLU's division has a branch, mlp_math.cuh) and the critical price's iterations; 0.69 ms
// without these two, of which the network alone takes 0.59 and the FP64 prices 0.64.  A third
// preparing warpgroup gives nothing (0.69 ms, 96 registers a thread) and costs small batches 8 %.
//
// Every wait is bounded; on a timeout the kernel sets *error, waits (bounded) for the MMAs in
// flight and frees its TMEM; the other side's waits then run out too.
#include <atomic>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "mlp.h"
#include "mlp_math.cuh"
#include "tc.cuh"
#include "tma.cuh"

namespace kwg {

namespace {

constexpr int kRows = 128;  // options per tile, one row per thread pair
constexpr int kNet = 2 * kRows;             // threads of the network's two warpgroups
constexpr int kSlots = 2;                   // warpgroups that prepare tiles, each with a slot
constexpr int kThreads = kNet + kSlots * kRows;
constexpr int kHalfCols = kMlpWidth / 2;  // accumulator columns per warpgroup
constexpr int kK1 = 16;     // layer-1 K: features hi 0..4, lo 5..9, zeros
constexpr uint32_t kW1Bytes = kMlpWidth * kK1 * 2;
constexpr uint32_t kWBytes = kMlpWidth * kMlpWidth * 2;
constexpr uint32_t kXBytes = kRows * kK1 * 2;
constexpr uint32_t kABytes = kRows * kMlpWidth * 2;
constexpr uint32_t kOffW1 = 0;
constexpr uint32_t kOffW = kOffW1 + kW1Bytes;  // W2, W3, W4
constexpr uint32_t kOffX = kOffW + 3 * kWBytes;
constexpr uint32_t kOffAhi = kOffX + kSlots * kXBytes;
constexpr uint32_t kOffAlo = kOffAhi + kABytes;
constexpr uint32_t kOffBias = kOffAlo + kABytes;            // 4 x 128 FP32
constexpr uint32_t kOffHead = kOffBias + 4 * kMlpWidth * 4;  // 128 FP32 (BF16 head weights, widened)
constexpr uint32_t kOffY = kOffHead + kMlpWidth * 4;         // 128 FP32: head partial sums
constexpr uint32_t kOffBase = kOffY + kRows * 4;             // kSlots x 128: base price, strike, floor
constexpr uint32_t kOffMisc = kOffBase + kSlots * kRows * 24;     // mbarriers, TMEM address
constexpr uint32_t kSmemBytes = kOffMisc + 128;
constexpr uint32_t kTmemCols = 256;  // two accumulators
static_assert(kSmemBytes <= 227 * 1024, "shared memory of an SM");
static_assert(kOffX % 1024 == 0 && kOffAhi % 1024 == 0 && kOffAlo % 1024 == 0, "operand tiles 1 KB aligned");

__device__ __forceinline__ void store_core(unsigned char* base, int kc, int row, int k, const __nv_bfloat16* v8)
{
    *reinterpret_cast<uint4*>(base + tc::core_offset(row, k, kc)) = *reinterpret_cast<const uint4*>(v8);
}

// Barrier of the network's threads, and whether `ok` holds in all of them.
__device__ __forceinline__ bool net_sync(bool ok)
{
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"((uint32_t)ok), "n"(kNet)
        : "memory");
    return all != 0;
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 1)
    mlp_price_fused(const kwg_option* __restrict__ opts, int n, MlpBox box, const __nv_bfloat16* __restrict__ wb,
                    const float* __restrict__ params, float y_scale, double* __restrict__ prices,
                    uint8_t* __restrict__ inside, int* __restrict__ error)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    const int tid = threadIdx.x, warp = tid / 32;
    const int row = tid % kRows, group = tid / kRows;
    uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + kOffMisc);  // MMAs of layer 1, of layers 2-4
    uint64_t* full = mbar + 2;       // [kSlots] a slot is written (one arrival per warp)
    uint64_t* empty = full + kSlots;  // [kSlots] a slot is consumed (one arrival per warp)
    uint32_t* tslot = reinterpret_cast<uint32_t*>(empty + kSlots);
    double* const slots = reinterpret_cast<double*>(sm + kOffBase);
    float* bias = reinterpret_cast<float*>(sm + kOffBias);
    float* head = reinterpret_cast<float*>(sm + kOffHead);
    float* ypart = reinterpret_cast<float*>(sm + kOffY);

    // resident weights: W1 = columns 0..15 of forward slot 0 ([128][64]); W2..W4 =
    // columns 0..127 of slots 1..3 ([128][256]); biases and the head row
    for (int v = tid; v < kMlpWidth * (kK1 / 8); v += blockDim.x) {
        const int row = v / (kK1 / 8), kq = v % (kK1 / 8);
        store_core(sm + kOffW1, kK1, row, kq * 8, wb + (size_t)row * kMlpInK + kq * 8);
    }
    for (int l = 0; l < 3; ++l) {
        const __nv_bfloat16* src = wb + (size_t)(l + 1) * kMlpFwdSlot;
        for (int v = tid; v < kMlpWidth * (kMlpWidth / 8); v += blockDim.x) {
            const int row = v / (kMlpWidth / 8), kq = v % (kMlpWidth / 8);
            store_core(sm + kOffW + l * kWBytes, kMlpWidth, row, kq * 8, src + (size_t)row * kMlpHidK + kq * 8);
        }
    }
    for (int i = tid; i < 4 * kMlpWidth; i += blockDim.x) bias[i] = params[kMlpWeights + i];
    for (int i = tid; i < kMlpWidth; i += blockDim.x) head[i] = __bfloat162float(wb[4 * kMlpFwdSlot + i]);
    const float head_b = params[kMlpWeights + 4 * kMlpWidth];
    if (warp == 0) {
        tc::tmem_alloc(smem_addr(tslot), kTmemCols);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) mbar_init(&mbar[b], 1);
        for (int b = 0; b < kSlots; ++b) {
            mbar_init(&full[b], kRows / 32);
            mbar_init(&empty[b], kRows / 32);
        }
        fence_mbar_init();
    }
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot;
    const int tiles = (n + kRows - 1) / kRows;
    bool ok = true;

    if (group >= 2) {
        // the CTA's tiles number slot, slot + kSlots, ... into this slot
        const int slot = group - 2;
        unsigned char* const xs = sm + kOffX + slot * kXBytes;
        double* const out = slots + slot * 3 * kRows + row;
        uint32_t phase = 0;
        for (int tile = blockIdx.x + slot * gridDim.x; tile < tiles && ok; tile += kSlots * gridDim.x, phase ^= 1u) {
            const int i = tile * kRows + row;
            float f[kMlpIn] = {0.f, 0.f, 0.f, 0.f, 0.f};
            double base = 0., strike = 0., least = 0.;
            if (i < n) {
                const kwg_option o = opts[i];
                const OptionTerms terms = option_terms(o);
                bool in = false;
                features(o, terms, box, f, in);
                base = base_price(o, terms);
                strike = o.k;
                least = o.e ? intrinsic(o) : NAN;  // fmax takes the other one
                if (inside) inside[i] = in ? 1 : 0;
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait(&empty[slot], phase ^ 1u));  // the first pass does not wait
            if (!ok) break;
            __align__(16) __nv_bfloat16 xr[kK1];
            split_features<kK1>(f, xr);
            store_core(xs, kK1, row, 0, xr);
            store_core(xs, kK1, row, 8, xr + 8);
            out[0] = base;
            out[kRows] = strike;
            out[2 * kRows] = least;
            tc::fence_proxy_async_smem();
            __syncwarp();
            if (tid % 32 == 0) mbar_arrive(&full[slot]);
        }
    } else {
        const int half = group;
        // this warp's 32 lanes (its rank in the warpgroup) and its warpgroup's columns
        const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * kHalfCols);
        const uint32_t idesc = tc::idesc_bf16_f32(kRows, kMlpWidth);
        const uint32_t sx = smem_addr(sm + kOffX), sw1 = smem_addr(sm + kOffW1), sw = smem_addr(sm + kOffW);
        const uint32_t shi = smem_addr(sm + kOffAhi), slo = smem_addr(sm + kOffAlo);
        bool pending1 = false, pending = false;  // MMAs in flight on mbar[0], mbar[1]
        uint32_t phase1 = 1, phase = 0;          // the last one issued on mbar[0], the next on mbar[1]

        // layer 1 of this CTA's it-th tile, from slot it % kSlots into the first accumulator
        auto layer1 = [&](int it) {
            const int slot = it % kSlots;
            if (!mbar_wait(&full[slot], (uint32_t)(it / kSlots) & 1u)) return false;
            tc::fence_after_sync();
            tc::mma_bf16(tmem, tc::smem_desc(sx + slot * kXBytes, 128, (kK1 / 8) * 128),
                         tc::smem_desc(sw1, 128, (kK1 / 8) * 128), idesc, false);
            tc::commit(smem_addr(&mbar[0]));
            phase1 ^= 1u;
            return true;
        };

        if (tid == 0 && (int)blockIdx.x < tiles) ok = pending1 = layer1(0);
        int it = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++it) {
            float y = 0.f;
            for (int l = 0; l < 4; ++l) {
                // a thread 0 that has not issued layer 1 lets the others' wait run out
                ok = ok && (l == 0 ? mbar_wait(&mbar[0], (uint32_t)it & 1u) : mbar_wait(&mbar[1], phase));
                if (l > 0) phase ^= 1u;
                ok = net_sync(ok);
                if (!ok) break;
                if (l == 0) pending1 = false;
                else pending = false;
                tc::fence_after_sync();
                const uint32_t acc = tl + (uint32_t)((l & 1) * kMlpWidth);
                if (l == 3) {
                    // the head in column order: columns 0..63, then 64..127 from that partial
                    float a[2][32];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int c = half * kHalfCols + 32 * h;
                        tc::tmem_ld32(acc + 32 * h, a[h]);
#pragma unroll
                        for (int j = 0; j < 32; ++j) a[h][j] = silu_f(a[h][j] + bias[3 * kMlpWidth + c + j]);
                    }
                    if (half == 1) {
                        net_sync(true);
                        y = ypart[row];
                    }
#pragma unroll
                    for (int j = 0; j < kHalfCols; ++j) y = fmaf(head[half * kHalfCols + j], a[j / 32][j % 32], y);
                    if (half == 0) {
                        ypart[row] = y;
                        net_sync(true);
                    }
                    break;
                }
#pragma unroll 1
                for (int cc = 0; cc < kHalfCols; cc += 32) {
                    const int c = half * kHalfCols + cc;  // the accumulator column
                    float v[32];
                    tc::tmem_ld32(acc + (uint32_t)cc, v);
                    __align__(16) __nv_bfloat16 hi[32], lo[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const float a = silu_f(v[j] + bias[l * kMlpWidth + c + j]);
                        hi[j] = __float2bfloat16(a);
                        lo[j] = __float2bfloat16(a - __bfloat162float(hi[j]));
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        store_core(sm + kOffAhi, kMlpWidth, row, c + 8 * q, hi + 8 * q);
                        store_core(sm + kOffAlo, kMlpWidth, row, c + 8 * q, lo + 8 * q);
                    }
                }
                // layer l + 2: activations (hi, then lo) x W_{l+2}
                tc::fence_proxy_async_smem();
                tc::fence_before_sync();
                net_sync(true);
                if (tid == 0) {
                    tc::fence_after_sync();
                    const uint32_t swl = sw + (uint32_t)l * kWBytes, dst = tmem + (uint32_t)((~l & 1) * kMlpWidth);
#pragma unroll
                    for (int kk = 0; kk < kMlpWidth / 16; ++kk)
                        tc::mma_bf16(dst, tc::smem_desc(shi + kk * 256, 128, (kMlpWidth / 8) * 128),
                                     tc::smem_desc(swl + kk * 256, 128, (kMlpWidth / 8) * 128), idesc, kk > 0);
#pragma unroll
                    for (int kk = 0; kk < kMlpWidth / 16; ++kk)
                        tc::mma_bf16(dst, tc::smem_desc(slo + kk * 256, 128, (kMlpWidth / 8) * 128),
                                     tc::smem_desc(swl + kk * 256, 128, (kMlpWidth / 8) * 128), idesc, true);
                    tc::commit(smem_addr(&mbar[1]));
                    // layer 3's epilogue has read the first accumulator: the next tile's layer 1
                    if (l == 2 && tile + (int)gridDim.x < tiles) ok = pending1 = layer1(it + 1);
                }
                pending = true;
            }
            if (!ok) break;
            if (half == 1) {
                const int slot = it % kSlots, i = tile * kRows + row;
                const double* const in = slots + slot * 3 * kRows + row;
                mbar_wait(&full[slot], (uint32_t)(it / kSlots) & 1u);  // complete: layer 1 has run on it
                const double v = in[0] + in[kRows] * (double)((y + head_b) / y_scale), least = in[2 * kRows];
                __syncwarp();
                if (tid % 32 == 0) mbar_arrive(&empty[slot]);
                if (i < n) prices[i] = fmax(v, least);
            }
            tc::fence_before_sync();  // TMEM reads of this tile precede the next tile's MMAs
        }
        if (!ok) {
            if (tid == 0 && error) atomicExch(error, 1);
            // let the MMAs in flight finish before TMEM is freed
            if (pending1) mbar_wait(&mbar[0], phase1);
            if (pending) mbar_wait(&mbar[1], phase ^ 1u);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, kTmemCols);
}

cudaError_t mlp_prepare_device()
{
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    if (const cudaError_t e = cudaGetDevice(&dev); e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load() & bit) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(mlp_price_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
    if (e == cudaSuccess) e = gemm_set_smem_limit();
    if (e == cudaSuccess) e = mlp_grad_set_smem_limit();
    if (e == cudaSuccess) done.fetch_or(bit);
    return e;
}

cudaError_t mlp_launch_price_fused(const kwg_option* opts, int n, const MlpBox& box, const __nv_bfloat16* wb,
                                   const float* params, float y_scale, double* prices, uint8_t* inside, int* error,
                                   int sms, cudaStream_t st)
{
    if (const cudaError_t e = mlp_prepare_device(); e != cudaSuccess) return e;
    const int tiles = (n + kRows - 1) / kRows;
    const int grid = tiles < sms ? tiles : sms;
    mlp_price_fused<<<grid, kThreads, kSmemBytes, st>>>(opts, n, box, wb, params, y_scale, prices, inside, error);
    return cudaGetLastError();
}

}  // namespace kwg
