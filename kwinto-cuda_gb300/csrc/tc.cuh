// tc.cuh -- inline-PTX wrappers for the 5th-generation tensor cores (tcgen05) and
// tensor memory (TMEM) on sm_100-family GPUs, as used by the MLP surrogate GEMMs.
//
// Conventions (kind::f16, cta_group::1, one CTA of 128 threads):
//   * A (M x K) and B (N x K) are BF16, K-major, staged in shared memory in the
//     no-swizzle "core matrix" layout: 8 rows x 16 bytes per core matrix (128 B,
//     rows contiguous); within a stage, core matrices run along K first.  The
//     descriptor's leading byte offset (LBO) is the distance between K-adjacent core
//     matrices, the stride byte offset (SBO) between M/N-adjacent ones.
//   * D (M x N, FP32) lives in TMEM: row i in lane i, column j in column j.
//   * One elected thread issues tcgen05.mma; tcgen05.commit arrives on an mbarrier
//     when the issued MMAs are complete; warps then read D with tcgen05.ld
//     (warp w of the CTA reads lanes 32w .. 32w+31).
#pragma once

#include <cstdint>

namespace kwg {
namespace tc {

// Shared-memory matrix descriptor, SWIZZLE_NONE: start address, LBO and SBO in
// 16-byte units, descriptor version 1 (bits 46-47), layout type 0 (bits 61-63).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Instruction descriptor for kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits
// 7-9 = 1, 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 in bits 17-22,
// M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int m, int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Instruction-descriptor bits: A, B in MN-major form.  The same core matrices (8 x 16 bytes) then hold
// 8 K-rows of 8 consecutive M or N elements; in the descriptor SBO stays the distance between
// core matrices adjacent along M or N, LBO the distance between those adjacent along K.
constexpr uint32_t kMajorMnA = 1u << 15, kMajorMnB = 1u << 16;

// Warp-collective TMEM allocation of `ncols` columns (power of 2, >= 32); the base
// address is written to shared memory at `dst`.
__device__ __forceinline__ void tmem_alloc(uint32_t dst_saddr, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_saddr), "r"(ncols)
                 : "memory");
}

__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T for one K-step (K = 16 for BF16).
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         bool accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

// Arrives once on the mbarrier when all MMAs issued so far by this thread complete.
__device__ __forceinline__ void commit(uint32_t mbar_saddr)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar_saddr)
                 : "memory");
}

__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Makes this thread's generic-proxy shared-memory writes visible to the tensor cores.
__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// 32 consecutive FP32 columns of this thread's TMEM lane (shape 32x32b, x32).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Byte offset of element (row, k) in a stage of `kc` BF16 columns laid out as
// core matrices [row/8][k/8] of 8 rows x 8 elements (LBO = 128 B along K,
// SBO = kc*16 B between 8-row groups).
__host__ __device__ constexpr uint32_t core_offset(int row, int k, int kc)
{
    return (uint32_t)(((row >> 3) * (kc >> 3) + (k >> 3)) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

}  // namespace tc
}  // namespace kwg
