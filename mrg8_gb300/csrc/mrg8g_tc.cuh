// mrg8g_tc.cuh -- the sm_103a instructions of the tensor-core kernel: shared
// memory barriers, bulk copies, tcgen05 products and tensor memory.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "mrg8g_device.cuh"

namespace mrg8g {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// A wait gives up after this long, or once another wait of its block has; each look
// at the barrier lasts at most about MRG8G_LOOK_NS.  A test sets both low.
#ifndef MRG8G_WAIT_LIMIT_NS
#define MRG8G_WAIT_LIMIT_NS 4000000000ull
#define MRG8G_LOOK_NS 1000000
#endif
constexpr unsigned long long kWaitLimitNs = MRG8G_WAIT_LIMIT_NS;

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.b32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "n"(MRG8G_LOOK_NS)
        : "memory");
    return ok != 0;
}

// Waits for the phase of `parity` to complete; false if it gave up, after
// setting the block's `gave_up` word (shared memory).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* gave_up) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (!mbar_try_wait(bar, parity)) {
        if (*gave_up) return false;
        if (global_ns() - t0 >= kWaitLimitNs) {
            *gave_up = 1;
            return false;
        }
    }
    return true;
}

// The last wait of a block that has given up, of phase 0: at most 4,000 looks.
__device__ __forceinline__ void mbar_wait_last(uint32_t bar) {
    for (int i = 0; i < 4000 && !mbar_try_wait(bar, 0); ++i) {
    }
}

// Bulk copy global -> shared, completing `bytes` on `bar` (16-byte aligned
// addresses and size).
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// Generic-proxy writes to shared memory become visible to the tensor cores.
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ------------------------------------------------------------ tensor memory

// All 32 lanes of one warp; the column address goes to *dst (shared memory).
__device__ __forceinline__ void tmem_alloc(uint32_t dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Four columns of the warp's 32 tensor-memory lanes, one lane per thread.
__device__ __forceinline__ void tmem_ld(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ------------------------------------------------------------------ products

// Shared-memory operand, K-major without swizzle: 16-byte K-chunks of eight
// rows contiguous, `chunk` bytes between K-chunks, `group` bytes between
// groups of eight rows.
__device__ __forceinline__ uint64_t tc_operand(uint32_t addr, uint32_t chunk, uint32_t group) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(chunk >> 4) << 16) | ((uint64_t)(group >> 4) << 32) |
           (1ull << 46);
}
// fp16 x fp16 -> fp32, both operands K-major, M = 128.
__host__ __device__ constexpr uint32_t tc_f16_desc(int n) { return (1u << 4) | ((uint32_t)(n / 8) << 17) | ((128u / 16) << 24); }

// One thread: D (+)= A B for 16 values of K.
__device__ __forceinline__ void tc_mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, bool add) {
    asm volatile(
        "{ .reg .pred p;\n\t"
        "setp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d),
        "l"(a), "l"(b), "r"(desc), "r"((uint32_t)add)
        : "memory");
}
// The thread's earlier products arrive on `bar` when they are complete.
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

}  // namespace mrg8g
