// Shared device-side helpers: step-buffer slots, the status word, bounded mbarrier waits, TMA and
// tcgen05 wrappers.  sm_100a only.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

namespace sgb {

// Step buffer slots (crates/sg-gpu/src/graph.rs:29-61).
enum : int { STEP_POS = 0, STEP_KV_LEN_SLIDING = 1, STEP_KV_LEN_GLOBAL = 2, STEP_Q0 = 3 };

// The sentinel the reference's shaders use instead of -inf (attn_decode_sliding.wgsl:77).
constexpr float NEG_SENTINEL = -3.0e38f;

// Device status word layout: word 0 = first error code (0 = none), word 1 = site id, word 2/3 = detail.
enum : uint32_t { DEV_OK = 0, DEV_ERR_TIMEOUT = 5, DEV_ERR_BOUNDS = 6 };

__device__ __forceinline__ void report_error(uint32_t* status, uint32_t code, uint32_t site, uint32_t a = 0,
                                             uint32_t b = 0)
{
    if (status != nullptr && atomicCAS(status, 0u, code) == 0u) {
        status[1] = site;
        status[2] = a;
        status[3] = b;
    }
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier ------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Every wait in this library is bounded: about a second of SM clock, after which the waiter
// records DEV_ERR_TIMEOUT with `site` and carries on (its results are then garbage, the host sees
// the error at the next sgb_sync).  A thread that has timed out once stops waiting altogether so
// that a broken pipeline drains in one bound, not one bound per stage.
constexpr long long WAIT_LIMIT_CYCLES = 2000000000LL;

// backoff_ns > 0 makes a waiter that is not latency-critical sleep between polls, leaving the issue
// slots to the warps that do the arithmetic.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t* status, uint32_t site, bool& failed,
                                          uint32_t backoff_ns = 0)
{
    if (failed) return false;
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
        if (backoff_ns) __nanosleep(backoff_ns);
        if (mbar_try_wait(bar, parity)) return true;
        if (clock64() - t0 > WAIT_LIMIT_CYCLES) {
            failed = true;
            report_error(status, DEV_ERR_TIMEOUT, site, blockIdx.x, parity);
            return false;
        }
    }
}

// The same by all lanes of a warp that leaves its loop when the wait has run out: they agree on it.  A limit that runs out in some
// lanes as the barrier completes for the others would send the first out of the loop and leave the rest at its next
// __syncwarp() for good.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, uint32_t* status, uint32_t site, bool& failed,
                                               uint32_t backoff_ns = 0)
{
    mbar_wait(bar, parity, status, site, failed, backoff_ns);
    failed = __any_sync(0xffffffffu, failed);
    return !failed;
}
// What a wait that ran out leaves in flight gets a bounded time to land before its target is handed to the next CTA.
__device__ __forceinline__ void let_copies_land()
{
    for (int i = 0; i < 50; i++) __nanosleep(1000);
}

// ---- TMA: every copy targets the issuing CTA only ---------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// Generic-proxy writes to shared memory made visible to the async proxy (TMA, tcgen05.mma).
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ---- tcgen05 / TMEM ------------------------------------------------------------------------------
// Waits without a limit until the SM has that many columns left, so it stands behind pdl_wait(): a CTA that held columns while
// it waited for its predecessor could hold those that a CTA of the predecessor still has to get.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols)
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
__device__ __forceinline__ void tc_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// MMAs and commits are issued by ONE thread, but the whole warp runs the issuing loop, with `one` set in the elected lane: the
// operands of tcgen05.mma are uniform registers, which the compiler computes in only where the code around them is uniform.  Moved there
// from a single thread's registers they cost that thread about 100 cycles an instruction, more than the tensor pipe needs for
// most: the int8 prefill took 521 us, in uniform code 346.
__device__ __forceinline__ uint32_t elect_one()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(e));
    return e;
}
// A value that is the same in all lanes, as one that the compiler knows to be.
template <typename T>
__device__ __forceinline__ T warp_uniform(T v) { return __shfl_sync(0xffffffffu, v, 0); }
// D[tmem] (+)= A[smem] * B[smem], f16 inputs, f32 accumulate.
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate, uint32_t one)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(one)
        : "memory");
}
// Same with the A operand in tensor memory: lane = row, each 32-bit column holds two consecutive
// f16 elements of K (so a K = 16 step spans 8 columns).
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate, uint32_t one)
{
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(one)
        : "memory");
}
// Arrive on an mbarrier once all tcgen05.mma issued so far by the elected thread have completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar, uint32_t one)
{
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n"
                 ::"r"(smem_u32(bar)), "r"(one)
                 : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp gets row (lane base + i).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
          "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
          "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
          "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}

// Shared-memory matrix descriptor for tcgen05.mma, 128-byte swizzle, version 1 (sm_100):
//   bits [0,14)  start address >> 4      bits [16,30) leading byte offset >> 4
//   bits [32,46) stride byte offset >> 4  bits [46,48) version = 1   bits [61,64) layout = 2 (SW128)
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor for kind::f16 with f16 A/B and f32 D:
//   [4,6) D format 1 = f32; [7,10) A format 0 = f16; [10,13) B format 0 = f16;
//   bit 15 A major (0 = K-major, 1 = MN-major); bit 16 B major; [17,23) N >> 3; [24,29) M >> 4.
__host__ __device__ constexpr uint32_t umma_idesc_f16(uint32_t m, uint32_t n, uint32_t a_mn_major, uint32_t b_mn_major)
{
    return (1u << 4) | (a_mn_major << 15) | (b_mn_major << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ unsigned long long globaltimer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// ---- small numeric helpers ------------------------------------------------------------------------
__device__ __forceinline__ float ex2(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Programmatic dependent launch: a kernel launched with the stream-serialization attribute may start while its
// predecessor in the stream still runs; it must call pdl_wait() before it touches anything the predecessor
// (or anything earlier in the stream) wrote.  pdl_launch_dependents() lets the successor's CTAs be scheduled as
// soon as every CTA of this grid has called it.  Both are no-ops for a plain launch.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Loads of what an earlier kernel of the stream may have written: not ld.global.nc, whose data has to be constant for as long as the
// kernel lives, and a kernel that starts before its predecessor has ended lives while that one still writes.  For the same
// reason no const pointer of such a kernel is __restrict__ (the compiler turns reads through one into ld.global.nc and may
// move them ahead of pdl_wait(); a volatile asm stays behind it).
template <typename T>
__device__ __forceinline__ T ld_global(const T* p)
{
    static_assert(sizeof(T) == 2 || sizeof(T) == 4 || sizeof(T) == 8 || sizeof(T) == 16, "one load");
    T v;
    if constexpr (sizeof(T) == 2) {
        uint16_t x;
        asm volatile("ld.global.b16 %0, [%1];" : "=h"(x) : "l"(p));
        memcpy(&v, &x, 2);
    } else if constexpr (sizeof(T) == 4) {
        uint32_t x;
        asm volatile("ld.global.b32 %0, [%1];" : "=r"(x) : "l"(p));
        memcpy(&v, &x, 4);
    } else if constexpr (sizeof(T) == 8) {
        uint2 x;
        asm volatile("ld.global.v2.b32 {%0, %1}, [%2];" : "=r"(x.x), "=r"(x.y) : "l"(p));
        memcpy(&v, &x, 8);
    } else {
        uint4 x;
        asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "l"(p));
        memcpy(&v, &x, 16);
    }
    return v;
}
// Barrier `id` (1..15; 0 is __syncthreads) over `threads` threads of the CTA, a multiple of 32.
__device__ __forceinline__ void named_barrier_sync(uint32_t id, uint32_t threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Barrier over `threads` threads that also tells every one of them whether `pred` held for any.
__device__ __forceinline__ bool named_barrier_or(uint32_t id, uint32_t threads, bool pred)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\t"
        "barrier.cta.red.or.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"(id), "r"(threads), "r"((uint32_t)pred)
        : "memory");
    return r != 0;
}
// Three-input maximum (one instruction on sm_100).
__device__ __forceinline__ float max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi)
{
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

}  // namespace sgb
