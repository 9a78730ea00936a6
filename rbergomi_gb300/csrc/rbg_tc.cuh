// rbg_tc.cuh -- sm_103a building blocks of the tensor-core kernels: bounded
// mbarrier waits, bulk copies, tcgen05 descriptors, MMA issue and commit.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace rbg {

constexpr int kTileM = 128;                  // MMA rows (TMEM lanes)
constexpr uint64_t kWaitNs = 2000000000ull;  // 2 s per wait

// ------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t globaltimer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Adds `bytes` to the phase's expected transaction count without arriving.
__device__ __forceinline__ void mbar_expect_tx_only(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Bulk copy global -> shared memory of this CTA (16-byte aligned addresses,
// a multiple of 16 bytes), completing `bytes` transactions on `bar`.
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Bulk copy shared memory of this CTA -> global (16-byte aligned addresses, a
// multiple of 16 bytes) as one bulk async-group of the issuing thread.
__device__ __forceinline__ void bulk_s2g(void* dst, uint32_t src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// The issuing thread's bulk stores: every source read (read0), every store
// complete (done0), or all but the most recent one complete (done1).
__device__ __forceinline__ void bulk_wait_read0() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_done0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_done1() { asm volatile("cp.async.bulk.wait_group 1;" ::: "memory"); }

// One wait attempt; the hardware may suspend the thread for up to 20 us
// (the suspend-time hint) until the phase completes, so waiting warps do not
// spin on the issue slots the working roles need.
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}

// Non-blocking test of a phase.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for the phase of the given parity; false on timeout or when
// another role already failed (then the caller winds down).  The error word
// and the clock are polled every 64 tries only (at most 64 x 20 us apart).  With `prof` set (diagnostic
// runs), lane 0 adds the cycles it waited to prof[site].  LIMIT_NS: the time
// limit, a compile-time constant (2 s in the pricing kernels).
template <uint64_t LIMIT_NS = kWaitNs>
static __device__ __noinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned int* err, unsigned int site,
                                       unsigned long long* prof = nullptr)
{
    if (mbar_try(bar, parity)) return true;
    const long long c0 = prof ? clock64() : 0;
    const uint64_t t0 = globaltimer();
    bool ok = true;
    for (uint32_t it = 1;; ++it) {
        if (mbar_try(bar, parity)) break;
        if ((it & 63u) == 0u) {
            if (*(volatile unsigned int*)err != 0u) { ok = false; break; }
            if (globaltimer() - t0 > LIMIT_NS) {
                atomicCAS(err, 0u, site);
                ok = false;
                break;
            }
        }
    }
    if (prof && (threadIdx.x & 31) == 0) atomicAdd(prof + site, (unsigned long long)(clock64() - c0));
    return ok;
}

// Waits up to 10 ms for a phase whatever the error word says: a CTA winding
// down after an error lets its own bulk copies in flight land before it exits.
static __device__ __noinline__ void mbar_drain(uint32_t bar, uint32_t parity)
{
    const uint64_t t0 = globaltimer();
    while (!mbar_try(bar, parity) && globaltimer() - t0 < 10000000ull) {
    }
}

// the same wait, made warp-uniform so .sync.aligned tcgen05 ops stay converged;
// the first try is inline, so a phase that has already completed (the common
// case in a balanced pipeline) costs no call
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, unsigned int* err, unsigned int site,
                                               unsigned long long* prof = nullptr)
{
    const bool ok = mbar_try(bar, parity) || mbar_wait(bar, parity, err, site, prof);
    return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// SW64 K-major shared-memory matrix descriptor (tcgen05 format): start
// address >> 4, LBO (unused for swizzled K-major) = 1, SBO = 8 rows x 64 B,
// version bit 46, layout type SWIZZLE_64B (4) in bits 61-63.
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t addr)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

// SW32 K-major descriptor for the 16-wide strip: 32-byte rows, SBO = 8 rows
// x 32 B, layout type SWIZZLE_32B (6).
__device__ __forceinline__ uint64_t sdesc_sw32(uint32_t addr)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(256 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)6 << 61);
}

// SW128 K-major descriptor for the TF32 A tile: 128-byte rows (32 FP32), SBO
// = 8 rows x 128 B, layout type SWIZZLE_128B (2).  A K = 8 step starts 32 B
// further into the row; the tile base is 1024-aligned, so the swizzle phase
// (address bits 7-9, the row) is unchanged and the base offset stays 0.
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t addr)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor, kind::tf32: D = F32, A = B = TF32 (2), both K-major.
__device__ __forceinline__ uint32_t idesc_tf32(int n)
{
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}

// FP32 -> TF32 rounded to nearest even (the low 13 bits of the result are 0).
__device__ __forceinline__ uint32_t tf32_rn(float x)
{
    uint32_t r;
    asm("cvt.rn.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// Instruction descriptor, kind::f16: D = F32, A = B = BF16 (1) or F16 (0),
// both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__device__ __forceinline__ uint32_t idesc_f16(int n, int ab_bf16)
{
    const uint32_t fmt = ab_bf16 ? 1u : 0u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

}  // namespace rbg
