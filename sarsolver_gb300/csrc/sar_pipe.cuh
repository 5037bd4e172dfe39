// sar_pipe.cuh -- device pieces the grid kernels share: check flags, pulse table loads, and the bounded
// mbarrier pipeline with 1-D bulk copies (sar_kernels.cu, sar_gather.cu, sar_scatter.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "sar_kernels.cuh"

namespace sar {

__device__ __forceinline__ void raise_flag(unsigned* flags, unsigned bit) {
    if (flags) atomicOr(flags, bit);
}

__device__ __forceinline__ PulseGeom load_pulse(const PulseGeom* p) {
    const float4* v = reinterpret_cast<const float4*>(p);
    const float4 a = __ldg(v), b = __ldg(v + 1), c = __ldg(v + 2), d = __ldg(v + 3);
    PulseGeom g;
    g.atx_hi[0] = a.x; g.atx_hi[1] = a.y; g.atx_hi[2] = a.z; g.atx_lo[0] = a.w;
    g.atx_lo[1] = b.x; g.atx_lo[2] = b.y; g.arx_hi[0] = b.z; g.arx_hi[1] = b.w;
    g.arx_hi[2] = c.x; g.arx_lo[0] = c.y; g.arx_lo[1] = c.z; g.arx_lo[2] = c.w;
    g.rref_hi = d.x; g.rref_lo = d.y; g.monostatic = d.z; g.pad = d.w;
    return g;
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_addr(bar))
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
                     smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
// Bounded wait for completion of the barrier phase with the given parity.  Between polls the
// warp sleeps with exponential backoff (first_ns doubling up to max_ns), so waiting warps leave
// the issue slots to the gathering warps and poll only a few times per wait; the wait gives up
// after `budget` clock cycles (kDefaultWaitBudgetCycles unless the launch sets its own).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned first_ns, unsigned max_ns,
                                          long long budget = kDefaultWaitBudgetCycles) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    unsigned ns = first_ns;
    while (true) {
        __nanosleep(ns);
        if (mbar_try_wait(bar, parity)) return true;
        if (clock64() - t0 > budget) return false;
        ns = min(2 * ns, max_ns);
    }
}
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// 1-D bulk copy global -> shared (16-byte aligned addresses, size a multiple of 16).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

}  // namespace sar
