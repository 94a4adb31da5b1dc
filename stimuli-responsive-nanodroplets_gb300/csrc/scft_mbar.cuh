/*
 * scft_mbar.cuh — the bounded mbarrier wait of the kernels that use asynchronous
 * copies or tensor-core products.
 */
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

/* Bounded wait for the mbarrier phase of the given parity: false after ~0.1 s.
 * CLUSTER: what completes the phase are stores of other CTAs of the cluster. */
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t mb, uint32_t parity)
{
    const long long t0 = clock64();
    for (;;) {
        uint32_t done;
        if (CLUSTER)
            asm volatile("{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P1, [%1], %2;\n\t"
                         "selp.b32 %0, 1, 0, P1;\n\t}"
                         : "=r"(done)
                         : "r"(mb), "r"(parity)
                         : "memory");
        else
            asm volatile("{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                         "selp.b32 %0, 1, 0, P1;\n\t}"
                         : "=r"(done)
                         : "r"(mb), "r"(parity)
                         : "memory");
        if (done) return true;
        if (clock64() - t0 > (1LL << 28)) return false;
    }
}
