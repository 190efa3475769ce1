// cluster.cuh -- exchange between the CTAs of one thread-block cluster (panel.cu, trsv.cu).
#pragma once
#include <stdint.h>

#include "waits.cuh"

namespace flg {

__device__ __forceinline__ uint32_t remote_addr(const void *p, int rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
// 8 bytes into CTA `rank`'s copy of *p, counted by its copy of the mbarrier
__device__ __forceinline__ void send(const void *p, const void *bar, int rank, unsigned long long v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(remote_addr(p, rank)),
                 "l"(v), "r"(remote_addr(bar, rank))
                 : "memory");
}
__device__ __forceinline__ void send(const void *p, const void *bar, int rank, double v) {
    send(p, bar, rank, (unsigned long long)__double_as_longlong(v));
}
__device__ __forceinline__ void expect_tx(const void *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ bool cluster_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded; after a timeout (the error word) every later wait gives up at once and the kernel runs to
// its end on garbage, which the host reports
__device__ __forceinline__ void cluster_wait(uint64_t *bar, uint32_t parity, int *err) {
    if (cluster_try_wait(bar, parity)) return;
    const unsigned long long t0 = global_ns();
    while (!cluster_try_wait(bar, parity)) {
        if (*(volatile int *)err) return;
        if (global_ns() - t0 > kWaitLimitNs) {
            atomicExch(err, 1);
            return;
        }
    }
}

}  // namespace flg
