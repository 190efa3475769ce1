// tc_common.cuh -- PTX wrappers shared by the tcgen05 kernels (tc_gemm.cu, slice_gemm.cu):
// mbarrier arrivals, 3-D TMA copies, shared-memory and instruction descriptors.
#pragma once
#include <cuda.h>
#include <stdint.h>

#include "waits.cuh"

namespace flg {

constexpr int TC_BM = 128;  // rows of an output tile (TMEM lanes)

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 3-D tiles: x (innermost, 16-byte aligned), row y, system z
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
        "[%2];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap *map, const void *src, int x, int y, int z) {
    asm volatile(
        "cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
            (uint64_t)map),
        "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sw128_desc(const void *p) {
    const uint64_t addr = smem_u32(p);
    uint64_t d = 0;
    d |= (addr >> 4) & 0x3FFFull;            // start address
    d |= (uint64_t)1 << 16;                  // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;        // stride byte offset: next 8-row group
    d |= (uint64_t)1 << 46;                  // descriptor version (tcgen05)
    d |= (uint64_t)2 << 61;                  // swizzle mode: 128B
    return d;
}

// instruction descriptor: D = F32, A/B format (TF32 = 2, BF16 = 1), K-major A and B, M = 128, N = bn
__host__ __device__ constexpr uint32_t tc_idesc(uint32_t fmt, int bn) {
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

// TMA operand map: nb systems (stride sb elements) of rows x K K-major elements (row stride ld_elems),
// box box_rows x 128 bytes x box_nb systems, 128B swizzle (tc_gemm.cu)
int make_operand_map(CUtensorMap *map, const void *base, int64_t rows, int64_t K, int64_t ld_elems, int mode,
                     int box_rows, int nb = 1, int64_t sb = 0, int box_nb = 1);

}  // namespace flg
