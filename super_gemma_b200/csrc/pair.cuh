// Two CTAs on one tensor-core tile (tcgen05 cta_group::2): a cluster of two, whose even CTA issues the MMAs of both.  A and D are
// half the rows of each CTA (M = 128: 64 rows a CTA, D's first N/2 columns in lanes 0..63 and the others in lanes 64..127 of the
// same tensor-memory columns), B is half its columns from each CTA's shared memory, at the same addresses in both.  Each
// CTA so loads half of what both read.  Cycles an instruction, f16, K = 16: N = 256 64, N = 128 45.
#pragma once

#include "sgb_common.cuh"

namespace sgb {

__device__ __forceinline__ uint32_t pair_rank()
{
    uint32_t r;
    asm("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}
// The same shared-memory address in the even CTA.
__device__ __forceinline__ uint32_t at_leader(const void* p)
{
    uint32_t out;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(out) : "r"(smem_u32(p)));
    return out;
}
__device__ __forceinline__ void pair_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on a barrier of the even CTA.  (With fences of cluster scope on both sides of every hand-over the int8 prefill took 705 us,
// without 451.)  It is for what lies in tensor memory or in this CTA's own shared memory and is read by this
// SM's half of the MMA that the barrier's waiter issues, after fence.proxy.async or tcgen05.fence on this side: neither side needs a
// fence of cluster scope.  Global memory is not handed over this way.
__device__ __forceinline__ void mbar_arrive_pair(uint32_t addr)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// A word of both CTAs' shared memory, there for all behind the next pair_sync().
__device__ __forceinline__ void store_both(uint32_t* p, uint32_t v)
{
    asm volatile(
        "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\tst.shared::cluster.u32 [a], %1;\n\t"
        "mapa.shared::cluster.u32 a, %0, 1;\n\tst.shared::cluster.u32 [a], %1;\n\t}"
        ::"r"(smem_u32(p)), "r"(v)
        : "memory");
}
// A copy into this CTA that reports to a barrier of the even CTA.
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* m, uint32_t bar_addr, int c0, int c1, int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_addr), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// Both CTAs allocate and free together.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D = A B, + D * 2^-DOWN with `accumulate`.
template <int DOWN = 0>
__device__ __forceinline__ void umma2_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate, uint32_t one)
{
    static_assert(DOWN >= 0 && DOWN <= 15, "scale-input-d");
    if constexpr (DOWN != 0)
        asm volatile(
            "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
            "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p, %6;\n\t}\n"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(one), "n"(DOWN)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
            "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
            ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(one)
            : "memory");
}
// Arrive on the barrier of both CTAs once all MMAs issued so far by this thread have completed.
__device__ __forceinline__ void umma2_commit(uint64_t* bar, uint32_t one)
{
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}\n"
        ::"r"(smem_u32(bar)), "h"((uint16_t)3), "r"(one)
        : "memory");
}

}  // namespace sgb
