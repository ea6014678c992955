// Shared-memory barriers and TMA copies (inline PTX, sm_90+ forms used on
// sm_103a), shared by the tensor-core filter and the staged projector.
// Every wait is bounded by the global timer, so a copy that never lands makes
// the caller give up instead of hanging.
#pragma once

#include <cstdint>

namespace ctk {
namespace tma {

// a wait gives up after this long (the waits of a healthy launch take microseconds)
constexpr unsigned long long kWaitNs = 1000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

// Makes barrier initialisation visible to the async (TMA) proxy; call after
// the inits, before the barrier's first use by another thread or a copy.
__device__ __forceinline__ void mbar_init_fence() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t a, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    return done != 0;
}

// Bounded wait on phase `parity`: false once `budget_ns` nanoseconds of the
// global timer have passed without the phase completing.  The timer is read
// only after 32 tries in vain: reading it for every wait took longer than the
// waits themselves.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          unsigned long long budget_ns = kWaitNs) {
    const uint32_t a = smem_u32(bar);
    for (int k = 0; k < 32; ++k)
        if (mbar_try(a, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 <= budget_ns)
        if (mbar_try(a, parity)) return true;
    return false;
}

// 1-D bulk copy global -> shared completing on `bar` (16-byte aligned
// addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

}  // namespace tma
}  // namespace ctk
