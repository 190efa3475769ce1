// slice_gemm.cu -- C -= A B in FP64 accuracy on the BF16 tensor cores (the Ozaki scheme).
//
//   C (m x nc, FP64, row-major, ldc)  -=  A (m x 64) * B (64 x nc)
//
// GB300 has two FP64 FMA lanes per SM and 64 times the FP32 lanes, while the BF16 tensor cores
// run three orders of magnitude above the FP64 pipe.  A and B come as eight 8-bit integer digits per
// value (slices.cuh), one BF16 slice per digit, each row of A and each column of B with its own
// exponent (K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication", Numer. Algorithms 59, 2012).
// The 36 slice products of order p = i + j <= 7 are exact integers below 2^24 and accumulate
// exactly in FP32 in TMEM, one accumulator per order; the epilogue joins the eight orders in
// 64-bit integers and rounds once to FP64 before the subtraction.  The dropped orders are below
// 2^-55 of (row maximum x column maximum) in the worst case, about 2^-61 in the mean: smaller
// than the rounding errors of a 64-term FP64 FMA chain (measured against 80-bit sums in
// tests/test_gpu_lu_f64.py).
//
// Persistent kernel, one CTA per SM (10 warps), each CTA a contiguous run of 128 x 32 tiles of C
// in row order, so that A's eight slices (128 KB) stay in shared memory over a row of tiles:
//   * warp 0 (one lane): TMA, A's block when the row changes, B's block (8 x 4 KB) into a
//     two-stage ring;
//   * warp 1 (one lane): 8 x 4 tcgen05.mma per tile (M = 128, K = 16) into one of two sets of eight
//     32-column accumulators (all 512 TMEM columns).  Slice q of A meets slices 0 .. 7 - q of B in one
//     instruction of N = 32 (8 - q): those slices follow one another in shared memory as the
//     orders' accumulators q .. 7 do in TMEM;
//   * warps 2-9: the epilogue of the other set, 16 columns per warp, the tile's C through a small
//     shared-memory transpose so that global accesses cover 64-byte row segments.
// What bounds it: the epilogue's latency (two warps per scheduler).  As 36 x 4 instructions of N = 32
// each read a slice of A for 32 columns, and with three FP64 operations per element to join the
// orders (the pipe has two lanes), a factorization took, n = 4,608 / 7,000, ms: 14.94 / 33.8; with the
// wide instructions 14.36 / 32.2; with the integer join as well 14.12 / 30.3.  Sixteen epilogue warps
// (15.0 / 33.8) or loads of C one chunk ahead (14.7 / 31.5) are slower.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "flg_common.cuh"
#include "slices.cuh"
#include "tc_common.cuh"
#include "waits.cuh"

namespace flg {

constexpr int SG_BN = 32, SG_THREADS = 320, SG_EPI_WARPS = 8;
constexpr int SG_A_SLICE = TC_BM * 128, SG_A_BYTES = kSlices * SG_A_SLICE;
constexpr int SG_B_SLICE = SG_BN * 128, SG_B_BYTES = kSlices * SG_B_SLICE;
constexpr int SG_STG_LD = 9;  // doubles per staged row of 8 columns
constexpr int SG_STG_BYTES = 32 * SG_STG_LD * 8;
constexpr size_t SG_SMEM = 1024 + SG_A_BYTES + 2 * SG_B_BYTES + SG_EPI_WARPS * SG_STG_BYTES;
static_assert(SG_SMEM <= 232448 - 256, "shared memory per CTA");

// eight consecutive TMEM columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr));
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// H + L 2^-32 for 64-bit integers below 2^62, rounded to a double by integer instructions: sign and magnitude,
// the top 64 of its 96 bits normalized, rounded to 53 (a tie away from zero).  As two conversions
// and an FMA it took three FP64 operations, 48 of the 64 clocks per 32 elements that the pipe needed.
__device__ __forceinline__ double join_orders(long long H, long long L) {
    const long long hi = H + (L >> 32);
    uint32_t w0 = (uint32_t)L, w1 = (uint32_t)hi, w2 = (uint32_t)((unsigned long long)hi >> 32);
    const uint32_t sign = w2 & 0x80000000u;
    if (sign)  // -(w2 w1 w0)
        asm("sub.cc.u32 %0, 0, %0;\n\tsubc.cc.u32 %1, 0, %1;\n\tsubc.u32 %2, 0, %2;" : "+r"(w0), "+r"(w1), "+r"(w2));
    int e = 1085;  // the exponent field, less one, for a leading bit at the top of w2
#pragma unroll
    for (int k = 0; k < 2; k++)
        if (w2 == 0) w2 = w1, w1 = w0, w0 = 0, e -= 32;
    const int lz = __clz((int)w2);
    const uint32_t m1 = __funnelshift_l(w1, w2, lz), m0 = __funnelshift_l(w0, w1, lz);
    const unsigned long long m = (unsigned long long)m1 << 32 | m0;
    const unsigned long long r = (m >> 11) + ((m0 >> 10) & 1) + ((unsigned long long)(uint32_t)(e - lz) << 52);
    const unsigned long long x = (w2 == 0 ? 0ull : r) | (unsigned long long)sign << 32;
    return __longlong_as_double((long long)x);
}
// t 2^e; the exponent field is added directly where neither side can leave the normal range
__device__ __forceinline__ double scale_pow2(double t, int e) {
    if (e > 900 || e < -900) return e >= kSliceNonFinite / 2 ? __longlong_as_double(0x7ff8000000000000ll) : scalbn(t, e);
    const int hi = __double2hiint(t);
    return (hi << 1) == 0 ? t : __hiloint2double(hi + e * (1 << 20), __double2loint(t));
}

__global__ void __launch_bounds__(SG_THREADS, 1) slice_update_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                     const __grid_constant__ CUtensorMap tmB,
                                                                     double *C, int64_t ldc, int m, int nc,
                                                                     const int *ea, const int *eb, int *err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem, *sB = smem + SG_A_BYTES, *stg = sB + 2 * SG_B_BYTES;
    __shared__ __align__(8) uint64_t afull, aempty, bfull[2], bempty[2], accf[2], acce[2], mma_done;
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntx = (nc + SG_BN - 1) / SG_BN, nty = (m + TC_BM - 1) / TC_BM;
    const int64_t ntiles = (int64_t)ntx * nty;
    const int64_t t0 = ntiles * blockIdx.x / gridDim.x, t1 = ntiles * (blockIdx.x + 1) / gridDim.x;
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) |
                               ((uint32_t)(TC_BM >> 4) << 24);  // FP32 accumulators, BF16, K-major, 128 x (N at bit 17)

    if (threadIdx.x == 0) {
        mbar_init(&afull, 1);
        mbar_init(&aempty, 1);
        for (int b = 0; b < 2; b++) {
            mbar_init(&bfull[b], 1);
            mbar_init(&bempty[b], 1);
            mbar_init(&accf[b], 1);
            mbar_init(&acce[b], SG_EPI_WARPS);
        }
        mbar_init(&mma_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t i = 0, na = 0;  // B loads and A loads issued
            int64_t row = -1;
            bool ok = true;
            for (int64_t t = t0; t < t1 && ok; t++, i++) {
                const int64_t rb = t / ntx, cb = t - rb * ntx;
                if (rb != row) {  // the MMAs of the previous row block release A
                    if (na > 0 && !mbar_wait(&aempty, (na & 1) ^ 1, err, kWaitLimitNs)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&afull, SG_A_BYTES);
                    tma_load_3d(sA, &tmA, &afull, 0, (int)(rb * TC_BM), 0);
                    na++;
                    row = rb;
                }
                const uint32_t s = i & 1, use = i >> 1;
                if (use > 0 && !mbar_wait(&bempty[s], (use & 1) ^ 1, err, kWaitLimitNs)) {
                    ok = false;
                    break;
                }
                mbar_expect_tx(&bfull[s], SG_B_BYTES);
                tma_load_3d(sB + s * SG_B_BYTES, &tmB, &bfull[s], 0, (int)(cb * SG_BN), 0);
            }
            // every load issued must have landed before the CTA exits
            if (na > 0) mbar_drain(&afull, (na - 1) & 1, err, kWaitLimitNs);
            for (uint32_t q = (i > 2 ? i - 2 : 0); q < i; q++) mbar_drain(&bfull[q & 1], (q >> 1) & 1, err, kWaitLimitNs);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t i = 0, na = 0;
            int64_t row = -1;
            for (int64_t t = t0; t < t1; t++, i++) {
                const int64_t rb = t / ntx;
                const uint32_t s = i & 1, use = i >> 1;
                if (use > 0 && !mbar_wait(&acce[s], (use & 1) ^ 1, err, kWaitLimitNs)) break;
                if (rb != row) {
                    if (!mbar_wait(&afull, na & 1, err, kWaitLimitNs)) break;
                    na++;
                    row = rb;
                }
                if (!mbar_wait(&bfull[s], use & 1, err, kWaitLimitNs)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d0 = tmem + s * (kSlices * SG_BN);
                const uint8_t *b0 = sB + s * SG_B_BYTES;
                // A's slice q meets B's slices 0 .. 7 - q at once: they lie one after the other like the orders'
                // accumulators q .. 7, so that N = 32 (8 - q) columns share one pass over A's slice
#pragma unroll
                for (int q = 0; q < kSlices; q++) {
                    const uint64_t ad = sw128_desc(sA + q * SG_A_SLICE), bd = sw128_desc(b0);
                    const uint32_t idesc = IDESC | ((uint32_t)((kSlices - q) * SG_BN >> 3) << 17);
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)  // 16 of the 64 K elements: 32 bytes of each row
                        asm volatile(
                            "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d0 + q * SG_BN),
                            "l"(ad + kk * 2), "l"(bd + kk * 2), "r"(idesc), "r"((q | kk) ? 1u : 0u)
                            : "memory");
                }
                mma_commit(&bempty[s]);
                mma_commit(&accf[s]);
                if (t + 1 == t1 || (t + 1) / ntx != rb) mma_commit(&aempty);
            }
            // every MMA issued has completed before the TMEM is freed
            mma_commit(&mma_done);
            mbar_drain(&mma_done, 0, err, kWaitLimitNs);
        }
    } else {
        const int q = warp & 3, h = (warp - 2) >> 2;  // TMEM lanes 32 q .. + 32, columns 16 h .. + 16
        double *st = (double *)(stg + (warp - 2) * SG_STG_BYTES);
        uint32_t i = 0;
        for (int64_t t = t0; t < t1; t++, i++) {
            const uint32_t s = i & 1, use = i >> 1;
            const int64_t rb = t / ntx, cb = t - rb * ntx;
            const int r0 = (int)(rb * TC_BM) + q * 32, c0 = (int)(cb * SG_BN) + h * 16;
            const int er = r0 + lane < m ? ea[r0 + lane] : 0;
            if (!__all_sync(0xffffffffu, mbar_wait(&accf[s], use & 1, err, kWaitLimitNs))) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int ch = 0; ch < 2; ch++) {
                const int cc = c0 + ch * 8;
                // the C elements of this chunk: lane covers column lane % 8 of rows lane / 8 + 4 k
                double cv[8];
                double *cp = C + (int64_t)(r0 + (lane >> 3)) * ldc + cc + (lane & 7);
                const bool cok = cc + (lane & 7) < nc;
#pragma unroll
                for (int k = 0; k < 8; k++)
                    cv[k] = cok && r0 + (lane >> 3) + 4 * k < m ? cp[(int64_t)4 * k * ldc] : 0.0;
                uint32_t v[kSlices][8];
                const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + s * (kSlices * SG_BN) + (uint32_t)(h * 16 + ch * 8);
#pragma unroll
                for (int p = 0; p < kSlices; p++) tmem_ld8(ta + p * SG_BN, v[p]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (ch == 1) {  // this warp has read its part of the accumulators
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce[s]);
                }
#pragma unroll
                for (int c = 0; c < 8; c++) {
                    int d[kSlices];
#pragma unroll
                    for (int p = 0; p < kSlices; p++) d[p] = __float2int_rn(__uint_as_float(v[p][c]));
                    // orders 0..3 in units of 2^-24 of the top order's, 4..7 in units of 2^-56
                    const long long H = (long long)(d[0] * 256 + d[1]) * 65536 + (d[2] * 256 + d[3]);
                    const long long L = (long long)(d[4] * 256 + d[5]) * 65536 + (d[6] * 256 + d[7]);
                    const double x = join_orders(H, L);
                    const int ec = cc + c < nc ? eb[cc + c] : 0;
                    st[lane * SG_STG_LD + c] = scale_pow2(x, er + ec - 36);
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const int r = (lane >> 3) + 4 * k;
                    if (cok && r0 + r < m) cp[(int64_t)4 * k * ldc] = cv[k] - st[r * SG_STG_LD + (lane & 7)];
                }
                __syncwarp();
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Slices of the rows of A (rows x 64, FP64, row stride lda): one warp per row, each lane two
// neighbouring elements, so every slice row is one 128-byte store.  S: [8][cap][64] BF16; e: [rows].
__global__ void __launch_bounds__(256) slice_rows_kernel(const double *A, int64_t lda, int64_t rows, int64_t cap,
                                                         __nv_bfloat16 *S, int *e) {
    const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= rows) return;
    const double x0 = A[r * lda + 2 * lane], x1 = A[r * lda + 2 * lane + 1];
    const int exmax = __reduce_max_sync(0xffffffffu, max(slice_exponent(x0), slice_exponent(x1)));
    const uint64_t w0 = slice_digits(x0, exmax), w1 = slice_digits(x1, exmax);
    if (lane == 0) e[r] = slice_scale(exmax);
    uint32_t *out = (uint32_t *)S + r * (kSliceK / 2) + lane;
#pragma unroll
    for (int k = 0; k < kSlices; k++)
        out[(int64_t)k * cap * (kSliceK / 2)] = __byte_perm(slice_bf16_hi(w0, k), slice_bf16_hi(w1, k), 0x7632);
}

int slice_rows(const double *A, int64_t lda, int64_t rows, int64_t cap, void *S, int *e, cudaStream_t st) {
    if (rows == 0) return FLG_OK;
    slice_rows_kernel<<<(unsigned)ceil_div(rows, 8), 256, 0, st>>>(A, lda, rows, cap, (__nv_bfloat16 *)S, e);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

// C (m x nc) -= A B from the slices SA (rows a0 .. a0 + m of [8][capA][64]) and SB (columns
// b0 .. b0 + nc of [8][capB][64]) with their exponents; err: device flag of a timed-out wait.
int slice_update(double *C, int64_t ldc, int64_t m, int64_t nc, const void *SA, int64_t capA, int64_t a0, const int *ea,
                 const void *SB, int64_t capB, int64_t b0, const int *eb, int *err, int max_ctas, cudaStream_t st) {
    if (m == 0 || nc == 0) return FLG_OK;
    FLG_REQUIRE(m < (1LL << 31) && nc < (1LL << 31), "bad slice update shape");
    CUtensorMap ma, mb;
    const __nv_bfloat16 *a = (const __nv_bfloat16 *)SA + a0 * kSliceK, *b = (const __nv_bfloat16 *)SB + b0 * kSliceK;
    FLG_TRY(make_operand_map(&ma, a, m, kSliceK, kSliceK, FLG_LU_BF16, TC_BM, kSlices, capA * kSliceK, kSlices));
    FLG_TRY(make_operand_map(&mb, b, nc, kSliceK, kSliceK, FLG_LU_BF16, SG_BN, kSlices, capB * kSliceK, kSlices));
    static bool attr_set = false;
    if (!attr_set) {
        FLG_CUDA(cudaFuncSetAttribute(slice_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SG_SMEM));
        attr_set = true;
    }
    const int64_t ntiles = ceil_div(m, TC_BM) * ceil_div(nc, SG_BN);
    const unsigned grid = (unsigned)std::min<int64_t>(ntiles, std::max(1, max_ctas));
    slice_update_kernel<<<grid, SG_THREADS, SG_SMEM, st>>>(ma, mb, C, ldc, (int)m, (int)nc, ea + a0, eb + b0, err);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

}  // namespace flg
