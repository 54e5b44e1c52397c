// tcgen05 building blocks in inline PTX: shared-memory descriptors, the integer MMA, its commit, fences and accumulator loads.
#pragma once
#include <stdint.h>

#include "abq_common.cuh"

namespace abq {

__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t smem_addr)
{
    // K-major operand tile, 128-byte rows, SWIZZLE_128B: 8-row groups are 1024 B apart (stride byte offset);
    // the leading byte offset is not used for swizzled K-major layouts (encoded as 1); descriptor version 1.
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3ffff) >> 4);       // start address, 16-byte units, bits [0,14)
    d |= (uint64_t)1 << 16;                            // leading byte offset (16 B units), bits [16,30)
    d |= (uint64_t)(1024 >> 4) << 32;                  // stride byte offset (16 B units), bits [32,46)
    d |= (uint64_t)1 << 46;                            // version (Blackwell), bits [46,48)
    d |= (uint64_t)2 << 61;                            // layout type SWIZZLE_128B, bits [61,64)
    return d;
}

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n"
                 ".reg .pred p;\n"
                 "setp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n"
                 "}\n" ::"r"(tmem_d),
                 "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive accumulator columns of this thread's TMEM lane, without the wait: several loads in flight, then one tmem_ld_wait()
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, int (&v)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                   "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// the same value into 16 consecutive accumulator columns (in pieces of four: a piece takes that many registers)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, int v)
{
#pragma unroll
    for (int c = 0; c < 16; c += 4)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %1, %1, %1};" ::"r"(taddr + c), "r"(v) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

} // namespace abq
