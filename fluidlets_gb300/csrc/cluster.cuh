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
}  // namespace flg
