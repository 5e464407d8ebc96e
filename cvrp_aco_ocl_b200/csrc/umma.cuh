// umma.cuh -- 5th-generation tensor-core (tcgen05) building blocks for sm_100a:
// tensor-memory allocation, shared-memory operand descriptors, the BF16 x BF16
// -> FP32 MMA issued by one thread, completion through an mbarrier, and
// accumulator reads.
//
// Operand tiles in shared memory.  A tile is R rows x 64 bf16 channels (R a
// multiple of 8), row r at 128 r bytes from a 1024-byte aligned start, and the
// 16-byte chunk j of a row (channels 8j..8j+7) stored at chunk j ^ (r mod 8):
// the 128-byte swizzle.  The same bytes are
//   * a K-major operand (M or N = rows, K = channels): stride-dimension byte
//     offset 1024 (next 8 rows), k-step s (16 channels) starts 32 s bytes in;
//   * an MN-major operand (M or N = channels, K = rows): stride-dimension byte
//     offset 1024 (next 8 rows of K), leading-dimension byte offset = the
//     distance of the next 64 channels, k-step s (16 rows) starts 2048 s bytes
//     in.
// A warp writes whole rows without bank conflicts.
//
// The descriptor and instruction-descriptor bit fields follow the PTX ISA
// description of tcgen05 matrix descriptors (start address >> 4 in bits 0-13,
// leading byte offset >> 4 in 16-29, stride byte offset >> 4 in 32-45,
// version 1 in 46-47, layout type 2 = 128-byte swizzle in 61-63) and of the
// kind::f16 instruction descriptor (D format F32 in bits 4-5, A and B format
// BF16 in 7-9 and 10-12, MN-major A and B in 15 and 16, N >> 3 in 17-22,
// M >> 4 in 24-28).
#pragma once

#include <cstdint>

#include "aco_device.cuh"

namespace aco {
namespace umma {

// Byte offset of 16-byte chunk j (channels 8j..8j+7) of row r.
__device__ __forceinline__ uint32_t sw_offset(int r, int j)
{
    return ((uint32_t)r << 7) + ((uint32_t)(j ^ (r & 7)) << 4);
}

constexpr uint64_t kDescSwizzle128 = (2ull << 61) | (1ull << 46) | ((uint64_t)(1024u >> 4) << 32);

// The tile at smem address `addr` read by rows (K-major), k-step s of its 64 channels.
__device__ __forceinline__ uint64_t desc_k(uint32_t addr, int s)
{
    return (uint64_t)(((addr + 32u * (uint32_t)s) >> 4) & 0x3FFFu) | (1ull << 16) | kDescSwizzle128;
}

// The tile at `addr` transposed (MN-major), k-step s of its rows; lbo: byte
// distance of the next 64 channels.
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr, int s, uint32_t lbo)
{
    return (uint64_t)(((addr + 2048u * (uint32_t)s) >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           kDescSwizzle128;
}

// Instruction descriptor: D F32, A/B BF16, M x N, either operand transposed (MN-major).
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, bool a_mn, bool b_mn)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ uint16_t bf16_bits(float x) // round to nearest even
{
    const __nv_bfloat16 b = __float2bfloat16_rn(x);
    return *reinterpret_cast<const uint16_t *>(&b);
}

// Tensor-memory allocation by one whole warp; the address lands in *slot.
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Generic-proxy shared-memory writes become visible to the tensor core (async proxy).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem]^T for one k-step; issued by a single thread.
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, bool acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
                 "l"(adesc), "l"(bdesc), "r"(idesc), "r"((uint32_t)acc)
                 : "memory");
}

// Arrive on the mbarrier once every MMA issued so far by this thread is done.
__device__ __forceinline__ void commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 consecutive fp32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
                   "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
                   "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// TMEM address of lane `lane`, column `col` relative to the allocation base.
__device__ __forceinline__ uint32_t taddr(uint32_t base, int lane, int col)
{
    return base + ((uint32_t)lane << 16) + (uint32_t)col;
}

} // namespace umma
} // namespace aco
