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
// 64-bit integers and rounds once to FP64 before the subtraction.  The dropped orders (seven products of
// 64 x 2^14 at 2^-76) are below 2^-53.2 of 2^(ea + eb), the scales of the row and the column, in the
// worst case and about 2^-59 of it for digits without a pattern.
//
// An FMA chain's error is small beside |C| and its own products instead.  Gaussian elimination in FP64
// of n unknowns promises n 2^-53 of |L||U| for every entry; the sliced sum keeps that, by a factor of
// four, where |C| is above 2^-(log2 n + 4) of 2^(ea + eb), or where some product is: where the near masks of the
// row and the column (slices.cuh) meet.  (A sum of products that are all zero is exact.)  The elements left
// over are recomputed in FP64 from L21 and U12 themselves: none of a random matrix, fewer than 1 in 10^5
// of a sphere's mobility matrix, all of a block whose 64 pivots differ in units.  With sliced sums
// everywhere a matrix with half its rows in units of 1e-20 of the others lost every digit of its solution.
//
// Persistent kernel, one CTA per SM (12 warps), each CTA a contiguous run of 128 x 32 tiles of C
// in row order, so that A's eight slices (128 KB) stay in shared memory over a row of tiles:
//   * warp 0 (one lane): TMA, A's block when the row changes, B's block (8 x 4 KB) into a
//     two-stage ring;
//   * warp 1 (one lane): 8 x 4 tcgen05.mma per tile (M = 128, K = 16) into one of two sets of eight
//     32-column accumulators (all 512 TMEM columns).  Slice q of A meets slices 0 .. 7 - q of B in one
//     instruction of N = 32 (8 - q): those slices follow one another in shared memory as the
//     orders' accumulators q .. 7 do in TMEM;
//   * warps 2-9: the epilogue of the other set, 16 columns per warp, the tile's C through a small
//     shared-memory transpose so that global accesses cover 64-byte row segments;
//   * warps 10-11: the masks, up to two tiles ahead of the epilogue: per column the rows that it leaves
//     open, in shared memory.
// Registers are limited to 128: the next panel's half_update and slice_rows need room beside a CTA of this kernel (at
// 168 a factorization of 4,608 unknowns took 14.7 ms).  The masks cost, n = 4,608 / 8,000 random 14.1 -> 14.3 /
// 41.8 -> 42.4 ms, sphere 14.0 -> 14.3 / 43.0 -> 45.4; a matrix whose rows all differ by tens of decades (every
// element recomputed on the FP64 pipe, as before there were slices) takes 80 ms at 4,608.
// What bounds it: the epilogue's latency (two warps per scheduler).  As 36 x 4 instructions of N = 32
// each read a slice of A for 32 columns, and with three FP64 operations per element to join the
// orders (the pipe has two lanes), a factorization took, n = 4,608 / 7,000, ms: 14.94 / 33.8; with the
// wide instructions 14.36 / 32.2; with the integer join as well 14.12 / 30.3.  Sixteen epilogue warps
// (15.0 / 33.8) or loads of C one chunk ahead (14.7 / 31.5) are slower.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "flg_common.cuh"
#include "slices.cuh"
#include "tc_common.cuh"
#include "waits.cuh"

namespace flg {

constexpr int SG_BN = 32, SG_EPI_WARPS = 8, SG_CHECK_WARPS = 2, SG_THREADS = 32 * (2 + SG_EPI_WARPS + SG_CHECK_WARPS);
constexpr int SG_BOUND = 512;  // threads that the registers would do for: 128 each
constexpr int SG_A_SLICE = TC_BM * 128, SG_A_BYTES = kSlices * SG_A_SLICE;
constexpr int SG_B_SLICE = SG_BN * 128, SG_B_BYTES = kSlices * SG_B_SLICE;
constexpr int SG_STG_LD = 9;  // doubles per staged row of 8 columns
constexpr int SG_FEW = 24;    // recomputed elements of a 32 x 8 chunk from which the whole chunk is
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

// The products A B (64 deep) in FP64 for flagged elements of a 32 x 8 chunk, into its staged sums st.  Bit k of a
// lane's flags: the element of row lane / 8 + 4 k, column lane % 8.  A: the chunk's first row, B: its first
// column (`rows` and `cols` of them exist).  Few elements: eight lanes each, four at a time; more: the
// whole chunk, a row per lane.
__device__ __noinline__ void exact_products(const double *A, const double *B, int64_t ld, int rows, int cols,
                                            unsigned flags, double *st) {
    const int lane = threadIdx.x & 31, grp = lane >> 3, l = lane & 7;
    if (__reduce_add_sync(0xffffffffu, __popc(flags)) >= SG_FEW) {
        const double *a = A + (int64_t)min(lane, rows - 1) * ld;
        double acc[8] = {};
#pragma unroll 1
        for (int q = 0; q < kSliceK; q += 2) {
            double av[2], bv[2][8];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                av[i] = a[q + i];
#pragma unroll
                for (int c = 0; c < 8; c++) bv[i][c] = B[(int64_t)(q + i) * ld + min(c, cols - 1)];
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int c = 0; c < 8; c++) acc[c] = fma(av[i], bv[i][c], acc[c]);
        }
#pragma unroll
        for (int c = 0; c < 8; c++) st[lane * SG_STG_LD + c] = acc[c];
        return;
    }
#pragma unroll 1
    for (int k = 0; k < 8; k++) {
        unsigned todo = __ballot_sync(0xffffffffu, flags >> k & 1);
        while (todo) {
            int e = -1;  // the lane that holds this group's element
#pragma unroll
            for (int q = 0; q < 4; q++) {
                e = q == grp && todo ? __ffs(todo) - 1 : e;
                todo &= todo - 1;
            }
            const int r = (e >> 3) + 4 * k, c = e & 7;
            double s = 0.0;
            if (e >= 0) {
                const double *a = A + (int64_t)r * ld + l, *b = B + (int64_t)l * ld + c;
                double av[8], bv[8];
#pragma unroll
                for (int q = 0; q < 8; q++) av[q] = a[8 * q], bv[q] = b[(int64_t)8 * q * ld];
#pragma unroll
                for (int q = 0; q < 8; q++) s = fma(av[q], bv[q], s);
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (e >= 0 && l == 0) st[r * SG_STG_LD + c] = s;
        }
    }
}

__global__ void __launch_bounds__(SG_BOUND, 1) slice_update_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                     const __grid_constant__ CUtensorMap tmB,
                                                                     double *C, int64_t ldc, int m, int nc,
                                                                     const double *A, const double *B, const int *ea,
                                                                     const int *eb, const SliceMask *ma, const SliceMask *mb,
                                                                     int near, int *err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem, *sB = smem + SG_A_BYTES, *stg = sB + 2 * SG_B_BYTES;
    __shared__ __align__(8) uint64_t afull, aempty, bfull[2], bempty[2], accf[2], acce[2], chkf[2], chke[2], mma_done;
    __shared__ unsigned s_apart[2][4][SG_BN], s_any[2][4];  // by 32 rows: a column's open rows, and the columns with any
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
            mbar_init(&chkf[b], SG_CHECK_WARPS);
            mbar_init(&chke[b], SG_EPI_WARPS);
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
    } else if (warp >= 2 + SG_EPI_WARPS) {
        const int w = warp - (2 + SG_EPI_WARPS);
        constexpr int G = 4 / SG_CHECK_WARPS;  // groups of 32 rows a warp
        const SliceMask all = make_uint4(~0u, ~0u, 0u, 0u);  // rows and columns beyond the matrix
        auto columns = [&](int64_t t) {
            const int col = (int)((t % ntx) * SG_BN) + lane;
            return t < t1 && col < nc ? mb[col] : all;
        };
        SliceMask mr[G], mn = columns(t0);
        int64_t rows_of = -1;
        uint32_t i = 0;
        for (int64_t t = t0; t < t1; t++, i++) {
            const uint32_t s = i & 1, use = i >> 1;
            const int64_t rb = t / ntx;
            const SliceMask mc = mn;
            mn = columns(t + 1);
            if (rb != rows_of) {
#pragma unroll
                for (int g = 0; g < G; g++) {
                    const int row = (int)(rb * TC_BM) + (w * G + g) * 32 + lane;
                    mr[g] = row < m ? ma[row] : all;
                }
                rows_of = rb;
            }
            if (use > 0 && !__all_sync(0xffffffffu, mbar_wait(&chke[s], (use & 1) ^ 1, err, kWaitLimitNs))) break;
#pragma unroll
            for (int g = 0; g < G; g++) {
                // columns that meet all 32 rows, in a value near all their maxima or by the number of them; the others
                const unsigned all_x = __reduce_and_sync(0xffffffffu, mr[g].x), all_y = __reduce_and_sync(0xffffffffu, mr[g].y);
                const int fewest = __reduce_min_sync(0xffffffffu, __popc(mr[g].x) + __popc(mr[g].y));
                const bool meets = ((mc.x & all_x) | (mc.y & all_y)) != 0 ||
                                   fewest + __popc(mc.x) + __popc(mc.y) > kSliceK;
                unsigned apart = 0;
                for (unsigned open = __ballot_sync(0xffffffffu, !meets); open; open &= open - 1) {
                    const int c = __ffs(open) - 1;
                    const unsigned nx = __shfl_sync(0xffffffffu, mc.x, c), ny = __shfl_sync(0xffffffffu, mc.y, c);
                    const unsigned zx = __shfl_sync(0xffffffffu, mc.z, c), zy = __shfl_sync(0xffffffffu, mc.w, c);
                    const unsigned a = __ballot_sync(0xffffffffu, ((mr[g].x & nx) | (mr[g].y & ny)) == 0 &&
                                                                      ((mr[g].z & zx) | (mr[g].w & zy)) != 0);
                    apart = lane == c ? a : apart;
                }
                const unsigned any = __ballot_sync(0xffffffffu, apart != 0);
                s_apart[s][w * G + g][lane] = apart;
                if (lane == 0) s_any[s][w * G + g] = any;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&chkf[s]);
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
            if (!__all_sync(0xffffffffu, mbar_wait(&accf[s], use & 1, err, kWaitLimitNs) &&
                                             mbar_wait(&chkf[s], use & 1, err, kWaitLimitNs)))
                break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned any = s_any[s][q] >> (16 * h) & 0xffffu;
            // the two chunks of this warp, in a usual tile without the branch to recomputed elements (with it everywhere,
            // 4,608 / 8,000 unknowns 14.5 / 44.8 ms and not 14.3 / 42.4)
            auto chunks = [&](auto open) {
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
                    if (decltype(open)::value && (any >> (ch * 8) & 0xffu)) {
                        const unsigned ap = s_apart[s][q][h * 16 + ch * 8 + (lane & 7)];
                        const int ec = cok ? eb[cc + (lane & 7)] : 0;
                        unsigned flags = 0;  // ... where C is small
#pragma unroll
                        for (int k = 0; k < 8; k++) {
                            const int r = (lane >> 3) + 4 * k;
                            if (ap >> r & 1 && cok && r0 + r < m &&
                                slice_exponent(cv[k]) - 1023 < ea[r0 + r] + ec - (2 * near + 2))
                                flags |= 1u << k;
                        }
                        if (__any_sync(0xffffffffu, flags)) {
                            exact_products(A + (int64_t)r0 * ldc, B + cc, ldc, m - r0, nc - cc, flags, st);
                            __syncwarp();
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const int r = (lane >> 3) + 4 * k;
                        if (cok && r0 + r < m) cp[(int64_t)4 * k * ldc] = cv[k] - st[r * SG_STG_LD + (lane & 7)];
                    }
                    __syncwarp();
                }
            };
            if (any) chunks(std::true_type{});
            else chunks(std::false_type{});
            if (lane == 0) mbar_arrive(&chke[s]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Slices of the rows of A (rows x 64, FP64, row stride lda): one warp per row, each lane two
// neighbouring elements, so every slice row is one 128-byte store.  S: [8][cap][64] BF16; e, mask: [rows].
__global__ void __launch_bounds__(256) slice_rows_kernel(const double *A, int64_t lda, int64_t rows, int64_t cap,
                                                         __nv_bfloat16 *S, int *e, SliceMask *mask, int near) {
    const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= rows) return;
    const double x0 = A[r * lda + 2 * lane], x1 = A[r * lda + 2 * lane + 1];
    const int exmax = __reduce_max_sync(0xffffffffu, max(slice_exponent(x0), slice_exponent(x1)));
    const uint64_t w0 = slice_digits(x0, exmax), w1 = slice_digits(x1, exmax);
    const unsigned near0 = __ballot_sync(0xffffffffu, slice_near(x0, exmax, near)),
                   near1 = __ballot_sync(0xffffffffu, slice_near(x1, exmax, near));
    const unsigned set0 = __ballot_sync(0xffffffffu, x0 != 0.0), set1 = __ballot_sync(0xffffffffu, x1 != 0.0);
    if (lane == 0) e[r] = slice_scale(exmax), mask[r] = make_uint4(near0, near1, set0, set1);
    uint32_t *out = (uint32_t *)S + r * (kSliceK / 2) + lane;
#pragma unroll
    for (int k = 0; k < kSlices; k++)
        out[(int64_t)k * cap * (kSliceK / 2)] = __byte_perm(slice_bf16_hi(w0, k), slice_bf16_hi(w1, k), 0x7632);
}

int slice_rows(const double *A, int64_t lda, int64_t rows, int64_t cap, void *S, int *e, SliceMask *mask, int near, cudaStream_t st) {
    if (rows == 0) return FLG_OK;
    slice_rows_kernel<<<(unsigned)ceil_div(rows, 8), 256, 0, st>>>(A, lda, rows, cap, (__nv_bfloat16 *)S, e, mask, near);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

// C (m x nc) -= A B: A (m x 64) and B (64 x nc) with C's row stride ldc, and their slices SA (rows 0 .. m of
// [8][capA][64]) and SB (columns b0 .. b0 + nc of [8][capB][64]) with exponents and masks; err: device flag
// of a timed-out wait.
int slice_update(double *C, int64_t ldc, int64_t m, int64_t nc, const double *A, const double *B, const void *SA,
                 int64_t capA, const int *ea, const SliceMask *ma, const void *SB, int64_t capB, int64_t b0, const int *eb,
                 const SliceMask *mb, int near, int *err, int max_ctas, cudaStream_t st) {
    if (m == 0 || nc == 0) return FLG_OK;
    FLG_REQUIRE(m < (1LL << 31) && nc < (1LL << 31), "bad slice update shape");
    CUtensorMap tma, tmb;
    const __nv_bfloat16 *b = (const __nv_bfloat16 *)SB + b0 * kSliceK;
    FLG_TRY(make_operand_map(&tma, SA, m, kSliceK, kSliceK, FLG_LU_BF16, TC_BM, kSlices, capA * kSliceK, kSlices));
    FLG_TRY(make_operand_map(&tmb, b, nc, kSliceK, kSliceK, FLG_LU_BF16, SG_BN, kSlices, capB * kSliceK, kSlices));
    FLG_ONCE_PER_DEVICE(
        FLG_CUDA(cudaFuncSetAttribute(slice_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)SG_SMEM)));
    const int64_t ntiles = ceil_div(m, TC_BM) * ceil_div(nc, SG_BN);
    const unsigned grid = (unsigned)std::min<int64_t>(ntiles, std::max(1, max_ctas));
    slice_update_kernel<<<grid, SG_THREADS, SG_SMEM, st>>>(tma, tmb, C, ldc, (int)m, (int)nc, A, B, ea, eb + b0,
                                                           ma, mb + b0, near, err);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

}  // namespace flg
