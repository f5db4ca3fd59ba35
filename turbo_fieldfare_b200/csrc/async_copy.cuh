// mbarrier and bulk asynchronous copy (cp.async.bulk) primitives shared by the kernels that stream weights
// through shared-memory rings. Every wait is bounded: a wait that runs out returns false and the caller records a
// device error code instead of hanging the GPU.
#pragma once

#include "tf_common.cuh"

namespace tf {

constexpr uint32_t kMbarSpinLimit = 1u << 21;

__device__ __forceinline__ uint32_t smem_addr_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier and bulk-copy primitives (all waits are bounded) ----
__device__ __forceinline__ void mbar_init(uint32_t addr, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(addr), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t addr) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" ::"r"(addr) : "memory");
}
// Hands a slot back after loads from it, once v, which depends on every one of them, is in a register: the barrier's address takes it, and a zero
// that the compiler cannot see (grids of one layer in z) takes it out again. A plain arrival waits for no load: neither for data that is still
// on its way nor for one that the compiler has moved to its first use behind the arrival (a tensor-core GEMM whose use was behind it had
// single rows with the weights of two stages later). An arrival behind stores of what was computed from the loads may be plain. (With two
// predicated arrivals, one for either outcome of a comparison of such values, steps of 11 to 200 tokens took 0.4 to 0.9 % longer.)
__device__ __forceinline__ void mbar_arrive_after(uint32_t addr, uint32_t v) {
    uint32_t zero;
    asm("mov.u32 %0, %%ctaid.z;" : "=r"(zero));
    mbar_arrive(addr | (v & zero));
}
__device__ __forceinline__ void mbar_arrive_after(uint32_t addr, float a, float b) { mbar_arrive_after(addr, __float_as_uint(a) | __float_as_uint(b)); }
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t addr, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }" ::"r"(addr), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity) {
    for (uint32_t i = 0; i < kMbarSpinLimit; ++i) {
        uint32_t ok;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// Both waits, the first one polled before the second in every round: what the second returns counts only once the first has
// passed, so the first may be what makes the second's parity unambiguous. The latencies of the two polls overlap.
__device__ __forceinline__ bool mbar_wait_both(uint32_t first, uint32_t first_parity, uint32_t second, uint32_t second_parity) {
    for (uint32_t i = 0; i < kMbarSpinLimit; ++i) {
        uint32_t ok;
        asm volatile("{ .reg .pred p, q; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; mbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4; "
                     "and.pred p, p, q; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok) : "r"(first), "r"(first_parity), "r"(second), "r"(second_parity) : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void bulk_copy_g2s(uint32_t smem_dst, const void* gmem_src, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_dst), "l"(gmem_src), "r"(bytes), "r"(mbar) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

}  // namespace tf
