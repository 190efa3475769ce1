// lu.cu -- dense LU factorizations and triangular solves.
//
// FP64 (the drop-in for scipy.linalg.solve, core/solve.py:64-67, and
// np.linalg.solve, swimming.py:101): right-looking blocked LU with partial
// pivoting, row-major storage, block width kPanel = 64.
//   cluster_panel     (panel.cu) panels of up to 8,192 rows, in two halves of 32
//                     columns on one 16-CTA cluster.
//   panel_f64_kernel  taller panels: cooperative launch over up to one CTA per SM; each CTA
//                     keeps a slab of panel rows in shared memory; one round of
//                     published candidates per column (pivot search is a
//                     grid-wide argmax, first index on ties as LAPACK's idamax),
//                     with the next column's look-ahead overlapping it.
//   swap_rows_kernel  the panel's row swaps on the columns left of it.
//   swap_trsm_kernel  the swaps and U12 = L11^-1 A12 right of it, and U12's BF16 slices.
//   slice_update      A22 -= L21 U12 in FP64 accuracy on the tensor cores (slice_gemm.cu).
//   trsv_cluster      (trsv.cu) the triangular solves of few right-hand sides.
//
// Low precision (preconditioner of FP64 GMRES-IR): blocked LU WITHOUT
// pivoting in FP32 storage, block FLG_LU_LOWP_BLOCK = 128: the diagonal block in
// the registers of one CTA, both panels by substitution in one launch, the
// trailing update on the tensor cores (tc_gemm.cu, deferred on two levels) or on
// CUDA cores (FLG_LU_FP32).  With the tensor cores the next diagonal block runs
// ahead on a side stream while the rest of each update finishes.  The inverses
// of the diagonal blocks' factors, kept in `dinv` for the solves, are one launch at the end.
//
// Every spin-wait (the panels' exchanges, the solves' dataflow, waits.cuh) is bounded and reports
// failure through a device flag instead of hanging.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "flg_common.cuh"
#include "panel.cuh"
#include "slices.cuh"
#include "trsv.cuh"
#include "waits.cuh"

namespace flg {

constexpr int kPanel = 64;                    // FP64 LU block width
constexpr int kNB = FLG_LU_LOWP_BLOCK;        // low-precision LU block

// ---- FP64 panel ------------------------------------------------------------------
// Partial-pivoting LU of the m x kb panel A[k0:n, k0:k0+kb] (LAPACK getf2's pivot
// choice: the largest |a| in the column, the first row on ties), one cooperative
// launch of up to one CTA per SM, each CTA holding `rpc` consecutive panel rows in
// shared memory (CTA c owns rows k0 + c rpc ...).  GB300 runs FP64 at ~2 FMA per
// SM and clock, so the panel's arithmetic must be spread over every SM; what
// limits it is the exchange between CTAs per column, which is kept to one
// round of published values:
//   * every CTA publishes, for column j, its candidate (the largest |a| among its
//     rows >= g, encoded with the column's parity bit in one 64-bit word released
//     after the candidate's full row and, by the owner of row g, row g itself);
//   * every CTA polls the words (acquire), picks the winner (largest value; on ties
//     the smaller CTA index, which owns the smaller rows), and reads the winning
//     row; the winner writes ipiv[g] and row g's old content into the pivot row,
//     the owner of g writes the pivot row into row g;
//   * look-ahead inside the panel: after scaling column j each CTA updates column
//     j + 1 first, finds its next candidate, completes the update of that row and
//     of row g + 1 and publishes them, and only then updates its other rows, so
//     the bulk of the rank-1 update overlaps the exchange.
// Every element receives the same fma, in the same column order, as in the
// textbook right-looking loop, so the factors do not depend on the CTA count.
// A word holds (bits(|a|) + 1) | parity << 63 (0 for "no rows >= g" or only
// NaN); the
// parity ((j >> 1) & 1) tells column j from column j - 2, which used the same
// one of the two buffers; the host presets both buffers to parity 1 before
// every panel.
struct PanelArgs {
    double *A;
    int64_t ld, n, k0;
    int kb, rpc;
    int32_t *ipiv;
    GridBar *bar;                 // err: a wait ran out; info: 1 + first zero pivot
    unsigned long long *word;     // [2][nblk]
    double *rowbuf;               // [2][nblk][kRowBufLd]: each CTA's candidate row and 1 / its pivot
    double *diagbuf;              // [2][kb]: row g
};

__device__ __forceinline__ void st_release_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

constexpr int kRowBufLd = kPanel + 8;  // a published row: kb values, then the reciprocal of its pivot

__global__ void __launch_bounds__(256) panel_f64_kernel(PanelArgs a) {
    extern __shared__ double P[];  // [rpc][kb]
    __shared__ double s_piv[kRowBufLd], s_old[kPanel];
    __shared__ unsigned long long red_w[8];
    __shared__ int red_c[8];
    __shared__ double s_rcp;  // 1 / this CTA's candidate value, published with its row
    __shared__ int s_win;     // winning CTA
    __shared__ int s_abort;
    const int nblk = gridDim.x, c = blockIdx.x, kb = a.kb, rpc = a.rpc;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int64_t r0 = a.k0 + (int64_t)c * rpc;
    const int nr = (int)max((int64_t)0, min((int64_t)rpc, a.n - r0));
    for (int e = t; e < nr * kb; e += blockDim.x) {
        const int lr = e / kb, j = e - lr * kb;
        P[e] = a.A[(r0 + lr) * a.ld + a.k0 + j];
    }
    if (t == 0) s_abort = 0;
    __syncthreads();

    // Local argmax of |P[., col]| over local rows >= lo (first row on ties), compared as
    // integers (the bits of a non-negative double order like its value; NaN never wins, as
    // in an FP comparison): the key bits(|a|) + 1 (0 if there is no candidate) and the local
    // row (-1), the same in every thread.  With `upd`, each row's column col first receives
    // its update from column col - 1 (multiplier P[., col - 1], pivot-row entry u).
    auto argmax = [&](int col, int lo, bool upd, double u, int &row) -> unsigned long long {
        unsigned long long best = 0;
        int brow = INT_MAX;
        for (int lr = lo + t; lr < nr; lr += blockDim.x) {
            double x = P[lr * kb + col];
            if (upd) {
                x = fma(-P[lr * kb + col - 1], u, x);
                P[lr * kb + col] = x;
            }
            const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
            const unsigned long long k = b > 0x7ff0000000000000ull ? 0ull : b + 1ull;
            if (k > best) {
                best = k;
                brow = lr;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int orow = __shfl_xor_sync(0xffffffffu, brow, o);
            if (ov > best || (ov == best && orow < brow)) {
                best = ov;
                brow = orow;
            }
        }
        if (lane == 0) {
            red_w[warp] = best;
            red_c[warp] = brow;
        }
        __syncthreads();
        unsigned long long bk = red_w[0];
        int br = red_c[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++)
            if (red_w[w] > bk || (red_w[w] == bk && red_c[w] < br)) {
                bk = red_w[w];
                br = red_c[w];
            }
        __syncthreads();
        row = bk == 0 ? -1 : br;
        return bk;
    };
    // the reciprocal of the candidate's value, computed while other threads work (one thread)
    auto candidate_rcp = [&](int col, int cand) {
        if (t == blockDim.x - 1) {
            const double v = cand >= 0 ? P[cand * kb + col] : 0.0;
            s_rcp = (v != 0.0 && isfinite(v)) ? 1.0 / v : 0.0;
        }
    };
    // publish column col's candidate (key k, local row cand, its reciprocal s_rcp) and, from
    // the owner, row g
    auto publish = [&](int col, unsigned long long k, int cand) {
        const int buf = col & 1;
        const unsigned long long par = (unsigned long long)((col >> 1) & 1) << 63;
        const int64_t g = a.k0 + col;
        double *rb = a.rowbuf + ((int64_t)buf * nblk + c) * kRowBufLd;
        if (cand >= 0 && t < kb) rb[t] = P[cand * kb + t];
        if (cand >= 0 && t == kb) rb[kPanel] = s_rcp;
        if (g >= r0 && g < r0 + nr && t < kb) a.diagbuf[buf * kb + t] = P[(g - r0) * kb + t];
        __syncthreads();  // the CTA's writes precede thread 0's release (cumulative through bar.sync)
        if (t == 0) st_release_u64(a.word + (int64_t)buf * nblk + c, par | k);
    };

    const int lo0 = (int)max((int64_t)0, min((int64_t)nr, a.k0 - r0));
    int mycand = -1;
    {
        const unsigned long long k0key = argmax(0, lo0, false, 0.0, mycand);
        candidate_rcp(0, mycand);
        __syncthreads();
        publish(0, k0key, mycand);
    }
    for (int j = 0; j < kb; j++) {
        const int64_t g = a.k0 + j;
        const int buf = j & 1;
        const unsigned long long par = (unsigned long long)((j >> 1) & 1);
        // (1) the winner of column j: every thread polls at most one CTA's word per pass
        //     (relaxed loads issued together, one acquire fence once all have arrived)
        {
            unsigned long long bv = 0;
            int bc = INT_MAX;
            for (int q0 = 0; q0 < nblk; q0 += blockDim.x) {
                const int q = q0 + t;
                if (q < nblk) {
                    const unsigned long long *w = a.word + (int64_t)buf * nblk + q;
                    unsigned long long u;
                    if (!wait_parity(w, par, u, kWaitLimitNs, &a.bar->err)) s_abort = 1;
                    const unsigned long long val = u & 0x7fffffffffffffffull;
                    if (val > bv) {
                        bv = val;
                        bc = q;
                    }
                }
            }
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long ov = __shfl_xor_sync(0xffffffffu, bv, o);
                const int oc = __shfl_xor_sync(0xffffffffu, bc, o);
                if (ov > bv || (ov == bv && oc < bc)) {
                    bv = ov;
                    bc = oc;
                }
            }
            if (lane == 0) {
                red_w[warp] = bv;
                red_c[warp] = bc;
            }
            __syncthreads();
            if (t == 0) {
                for (int w = 1; w < (int)(blockDim.x >> 5); w++)
                    if (red_w[w] > red_w[0] || (red_w[w] == red_w[0] && red_c[w] < red_c[0])) {
                        red_w[0] = red_w[w];
                        red_c[0] = red_c[w];
                    }
                s_win = red_c[0];
            }
        }
        __syncthreads();
        if (s_abort) return;
        // no candidate anywhere (every |a| of the column NaN): row g stays, as the pivot
        const bool none = s_win == INT_MAX;
        const int own_g = (int)((g - a.k0) / rpc);
        const int win = none ? own_g : s_win;
        // (2) the pivot row with its reciprocal, and for the winner the old row g
        if (t <= kb) {
            if (none) s_piv[t] = t < kb ? __ldcg(a.diagbuf + buf * kb + t) : 0.0;
            else s_piv[t == kb ? kPanel : t] = __ldcg(a.rowbuf + ((int64_t)buf * nblk + win) * kRowBufLd +
                                                      (t == kb ? kPanel : t));
            if (win == c && t < kb) s_old[t] = __ldcg(a.diagbuf + buf * kb + t);
        }
        __syncthreads();
        // (3) the swap
        const int64_t p = (win == c) ? (none ? g : r0 + mycand) : -1;
        if (win == c && t == 0) a.ipiv[g] = (int32_t)p;
        if (t < kb) {
            if (win == c && p != g) P[(p - r0) * kb + t] = s_old[t];
            if (g >= r0 && g < r0 + nr) P[(g - r0) * kb + t] = s_piv[t];
        }
        const int lr1 = (int)max((int64_t)0, min((int64_t)nr, g + 1 - r0));  // first local row > g
        const double piv = s_piv[j];
        const bool ok = piv != 0.0 && isfinite(piv);
        if (!ok && t == 0) atomicCAS(&a.bar->info, 0, (int)(g + 1));
        // (3b) scale column j below g (rows > g are not touched by the swap's writes to row g;
        //      the winner's write to row p is by the same threads, t < kb, before their scaling)
        __syncthreads();
        if (ok) {
            const double rp = s_piv[kPanel];  // = 1 / piv, computed by the publisher
            for (int lr = lr1 + t; lr < nr; lr += blockDim.x) P[lr * kb + j] *= rp;
        }
        __syncthreads();
        if (j + 1 == kb) break;
        // (4) look-ahead: column j + 1 (updated on the way), the next candidate, its row and
        //     row g + 1, published
        int cand;
        const unsigned long long v = argmax(j + 1, lr1, ok, s_piv[j + 1], cand);
        candidate_rcp(j + 1, cand);
        const int lg1 = (g + 1 >= r0 && g + 1 < r0 + nr) ? (int)(g + 1 - r0) : -1;
        if (ok) {
            const int q = j + 2 + (t & 63);
            const int which = t >> 6;  // 0: the candidate row, 1: row g + 1
            const int lr = which == 0 ? cand : (lg1 != cand ? lg1 : -1);
            if (which < 2 && lr >= 0 && q < kb) P[lr * kb + q] = fma(-P[lr * kb + j], s_piv[q], P[lr * kb + q]);
        }
        __syncthreads();
        publish(j + 1, v, cand);
        // (5) the rest of the rank-1 update (columns > j + 1), beside the exchange
        if (ok) {
            const int q = t % kPanel, rg = t / kPanel;
            constexpr int kRowStep = 256 / kPanel;
            if (q > j + 1 && q < kb) {
                const double u = s_piv[q];
                for (int lr = lr1 + rg; lr < nr; lr += kRowStep)
                    if (lr != cand && lr != lg1) P[lr * kb + q] = fma(-P[lr * kb + j], u, P[lr * kb + q]);
            }
        }
        mycand = cand;
        __syncthreads();
    }
    for (int e = t; e < nr * kb; e += blockDim.x) {
        const int lr = e / kb, j = e - lr * kb;
        a.A[(r0 + lr) * a.ld + a.k0 + j] = P[e];
    }
}

// ---- row interchanges and U12 ---------------------------------------------------------
// The net effect of a panel's kb <= 64 row interchanges (LAPACK laswp: for q = 0..kb-1 swap rows
// k0 + q and ipiv[k0 + q]) on at most 2 kb rows: slot q < 64 is row k0 + q, slot 64 + q the pivot
// row ipiv[k0 + q] where it lies below the panel and no earlier q named it.  dst[slot] is the
// slot's row (-1: unused), src[slot] the row whose old content it receives, found by running
// the interchanges backwards from the slot's row; one thread per slot, 64 dependent
// compare-selects instead of 64 dependent swaps.
__device__ __forceinline__ void swap_slots(const int32_t *ipiv, int64_t k0, int kb, int *piv, int *dst, int *src) {
    for (int q = threadIdx.x; q < kPanel; q += blockDim.x) piv[q] = q < kb ? ipiv[k0 + q] : -1;
    __syncthreads();
    for (int s = threadIdx.x; s < 2 * kPanel; s += blockDim.x) {
        const int q = s & (kPanel - 1);
        int r = q < kb ? (int)k0 + q : -1;
        if (s >= kPanel && q < kb) {
            r = piv[q] >= (int)k0 + kb ? piv[q] : -1;
            for (int p = 0; p < q; p++) r = piv[p] == r ? -1 : r;
        }
        dst[s] = r;
        for (int p = kb - 1; p >= 0; p--) {
            const int a = (int)k0 + p, b = piv[p];
            r = r == a ? b : r == b ? a : r;
        }
        src[s] = r;
    }
    __syncthreads();
}

// the interchanges alone, on the columns [c0, c1): four lanes per column, each gathering its 32
// slots with independent loads before any lane of the column writes
constexpr int kSwapThreads = 128, kSwapCols = kSwapThreads / 4;
__global__ void __launch_bounds__(kSwapThreads) swap_rows_kernel(double *A, int64_t ld, const int32_t *ipiv, int64_t k0,
                                                                 int kb, int64_t c0, int64_t c1) {
    __shared__ int piv[kPanel], dst[2 * kPanel], src[2 * kPanel];
    swap_slots(ipiv, k0, kb, piv, dst, src);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 3;
    const int64_t c = c0 + (int64_t)blockIdx.x * kSwapCols + warp * 8 + (lane & 7);
    constexpr int R = 2 * kPanel / 4;
    double x[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int s = 4 * i + g;
        if (c < c1 && dst[s] >= 0 && dst[s] != src[s]) x[i] = A[src[s] * ld + c];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int s = 4 * i + g;
        if (c < c1 && dst[s] >= 0 && dst[s] != src[s]) A[dst[s] * ld + c] = x[i];
    }
}

// The interchanges and U12 = L11^-1 A12 (unit lower L11 = A[k0:k0+64, k0:k0+64]) on the columns
// [c0, c1) right of a full panel, and the slices of U12's columns for the trailing update
// (slices.cuh): SB [8][cap][64] BF16 with column c at row c - c0, exponents and masks eb, mb[c - c0].  G lanes per
// column, lane group g holding rows G i + g: the substitution runs column by column of L11
// (every row's FMAs in the same order as row by row, but independent of one another).  An FP64
// warp instruction takes 64 clocks of its scheduler, so a warp's 544 (G = 4) or 160 (G = 16) of them
// are the kernel's time: 16 lanes per column spread the few hundred columns of a small system over all
// schedulers, 4 waste fewer FMAs on rows already solved where there are columns for every
// scheduler anyway.  `warps` of a CTA's eight have columns; all load L11 and work out the
// interchanges.  Two CTAs per SM (128 registers): the wide launch beside a cluster panel has more
// CTAs than SMs left (one per SM: 14.8 ms for 4,608 unknowns, two: 14.7).
constexpr int kTrsmThreads = 256, kTrsmWarps = kTrsmThreads / 32;
constexpr int kTrsmStgLd = kPanel + 8;              // 16-bit words per staged slice row (no bank conflicts)
constexpr size_t trsm_smem(int G, int warps) {
    return sizeof(double) * kPanel * kPanel + sizeof(uint16_t) * kSlices * (32 / G) * kTrsmStgLd * warps;
}
template <int G>
__global__ void __launch_bounds__(kTrsmThreads, 2) swap_trsm_kernel(double *A, int64_t ld, const int32_t *ipiv, int64_t k0,
                                                                 int64_t c0, int64_t c1, int warps, uint16_t *SB,
                                                                 int64_t cap, int *eb, SliceMask *mb, int near_range) {
    extern __shared__ __align__(16) double Lt[];  // [64][64]: Lt[q][r] = L11[r][q]; then the warps' staged slices
    __shared__ int piv[kPanel], dst[2 * kPanel], src[2 * kPanel];
    constexpr int COLS = 32 / G, R = kPanel / G;  // columns per warp, rows per lane
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane / COLS, cl = lane % COLS;
    {  // (swizzled rows: no bank conflicts either way)
        double v[kPanel * kPanel / kTrsmThreads];
#pragma unroll
        for (int k = 0; k < kPanel * kPanel / kTrsmThreads; k++) {
            const int e = threadIdx.x + k * kTrsmThreads;
            v[k] = A[(k0 + e / kPanel) * ld + k0 + e % kPanel];
        }
#pragma unroll
        for (int k = 0; k < kPanel * kPanel / kTrsmThreads; k++) {
            const int e = threadIdx.x + k * kTrsmThreads, r = e / kPanel, q = e % kPanel;
            Lt[q * kPanel + (r ^ (q & 15))] = v[k];
        }
    }
    swap_slots(ipiv, k0, kPanel, piv, dst, src);
    const int64_t cw = c0 + ((int64_t)blockIdx.x * warps + warp) * COLS;
    if (warp >= warps || cw >= c1) return;
    const bool live = cw + cl < c1;
    const int64_t c = live ? cw + cl : c1 - 1;
    double x[R], y[R];
#pragma unroll
    for (int i = 0; i < R; i++) x[i] = A[src[G * i + g] * ld + c];
#pragma unroll
    for (int i = 0; i < R; i++)
        if (dst[kPanel + G * i + g] >= 0) y[i] = A[src[kPanel + G * i + g] * ld + c];
    __syncwarp();  // every lane of a column has read before any writes
#pragma unroll
    for (int i = 0; i < R; i++)
        if (live && dst[kPanel + G * i + g] >= 0) A[dst[kPanel + G * i + g] * ld + c] = y[i];
#pragma unroll
    for (int q = 0; q < kPanel - 1; q++) {
        const double xq = __shfl_sync(0xffffffffu, x[q / G], (q % G) * COLS + cl);
        const double *l = Lt + q * kPanel;
#pragma unroll
        for (int i = q / G; i < R; i++) {
            const double v = fma(-l[(G * i + g) ^ (q & 15)], xq, x[i]);
            x[i] = (i > q / G || g > q % G) ? v : x[i];
        }
    }
    int exmax = 1;
#pragma unroll
    for (int i = 0; i < R; i++) {
        if (live) A[(k0 + G * i + g) * ld + c] = x[i];
        exmax = max(exmax, slice_exponent(x[i]));
    }
#pragma unroll
    for (int o = COLS; o < 32; o <<= 1) exmax = max(exmax, __shfl_xor_sync(0xffffffffu, exmax, o));
    if (live && g == 0) eb[c - c0] = slice_scale(exmax);
    {  // this lane's rows have the parity of g, so their bits lie in one word of each mask
        unsigned near = 0, set = 0;
#pragma unroll
        for (int i = 0; i < R; i++) {
            const unsigned bit = 1u << ((G * i + g) >> 1);
            near |= slice_near(x[i], exmax, near_range) ? bit : 0u;
            set |= x[i] != 0.0 ? bit : 0u;
        }
#pragma unroll
        for (int o = 2 * COLS; o < 32; o <<= 1) {
            near |= __shfl_xor_sync(0xffffffffu, near, o);
            set |= __shfl_xor_sync(0xffffffffu, set, o);
        }
        if (live && g < 2) {
            unsigned *w = reinterpret_cast<unsigned *>(mb + (c - c0)) + g;
            w[0] = near, w[2] = set;
        }
    }
    uint16_t *stg = (uint16_t *)(Lt + kPanel * kPanel) + warp * (kSlices * COLS * kTrsmStgLd);
#pragma unroll
    for (int i = 0; i < R; i++) {
        const uint64_t w = slice_digits(x[i], exmax);
#pragma unroll
        for (int k = 0; k < kSlices; k++)
            stg[(k * COLS + cl) * kTrsmStgLd + G * i + g] = (uint16_t)(slice_bf16_hi(w, k) >> 16);
    }
    __syncwarp();
    // the staged rows (slice, column) of 128 bytes: eight lanes per row
#pragma unroll
    for (int it = 0; it < kSlices * COLS / 4; it++) {
        const int row = it * 4 + (lane >> 3), k = row / COLS, col = row % COLS, ch = (lane & 7) * 8;
        if (cw + col < c1)
            *reinterpret_cast<uint4 *>(SB + ((int64_t)k * cap + (cw + col - c0)) * kSliceK + ch) =
                *reinterpret_cast<const uint4 *>(stg + row * kTrsmStgLd + ch);
    }
}
constexpr int kTrsmWide = 2 * 8;
static int swap_trsm(double *A, int64_t ld, const int32_t *ipiv, int64_t k0, int64_t c0, int64_t c1, uint16_t *SB,
                     int64_t cap, int *eb, SliceMask *mb, int near, cudaStream_t st) {
    const int64_t nc = c1 - c0;
    FLG_ONCE_PER_DEVICE(
        FLG_CUDA(cudaFuncSetAttribute(swap_trsm_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)trsm_smem(4, kTrsmWarps)));
        FLG_CUDA(cudaFuncSetAttribute(swap_trsm_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)trsm_smem(16, kTrsmWarps))));
    // G = 4 once its warps (8 columns each) fill half of the schedulers; below, G = 16's shorter chain
    const bool wide = nc >= kTrsmWide * (int64_t)sm_count();
    const int cols = wide ? 8 : 2;
    const int w = (int)std::min<int64_t>(kTrsmWarps, ceil_div(nc, (int64_t)cols * sm_count()));
    const unsigned grid = (unsigned)ceil_div(nc, (int64_t)w * cols);
    if (wide) swap_trsm_kernel<4><<<grid, kTrsmThreads, trsm_smem(4, w), st>>>(A, ld, ipiv, k0, c0, c1, w, SB, cap, eb, mb, near);
    else swap_trsm_kernel<16><<<grid, kTrsmThreads, trsm_smem(16, w), st>>>(A, ld, ipiv, k0, c0, c1, w, SB, cap, eb, mb, near);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

// the trailing update on the tensor cores (slice_gemm.cu)
int slice_rows(const double *A, int64_t lda, int64_t rows, int64_t cap, void *S, int *e, SliceMask *mask, int near,
               cudaStream_t st);
int slice_update(double *C, int64_t ldc, int64_t m, int64_t nc, const double *A, const double *B, const void *SA,
                 int64_t capA, const int *ea, const SliceMask *ma, const void *SB, int64_t capB, int64_t b0, const int *eb,
                 const SliceMask *mb, int near, int *err, int max_ctas, cudaStream_t st);

// ---- FP64 triangular solves (getrs) ------------------------------------------------
// Row interchanges in LAPACK order (swap rows r and ipiv[r] for r = 0, 1, ...).
// One CTA per right-hand side column; the column sits in shared memory while one
// thread applies the swaps (they compose, so they are sequential), then goes back.
constexpr int kPivSmemMax = 24576;  // doubles (192 KB)
__global__ void __launch_bounds__(256) apply_pivots_smem_kernel(double *B, int64_t ldb, const int32_t *ipiv,
                                                                int64_t n) {
    extern __shared__ double col[];
    const int64_t c = blockIdx.x;
    for (int64_t r = threadIdx.x; r < n; r += blockDim.x) col[r] = B[r * ldb + c];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int64_t r = 0; r < n; r++) {
            const int64_t p = ipiv[r];
            if (p != r) {
                const double t = col[r];
                col[r] = col[p];
                col[p] = t;
            }
        }
    }
    __syncthreads();
    for (int64_t r = threadIdx.x; r < n; r += blockDim.x) B[r * ldb + c] = col[r];
}
// the same for columns too long for shared memory (one thread per column, global memory)
__global__ void apply_pivots_kernel(double *B, int64_t ldb, int64_t nrhs, const int32_t *ipiv, int64_t n) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nrhs) return;
    for (int64_t r = 0; r < n; r++) {
        const int64_t p = ipiv[r];
        if (p != r) {
            const double t = B[r * ldb + c];
            B[r * ldb + c] = B[p * ldb + c];
            B[p * ldb + c] = t;
        }
    }
}

// solve the diagonal block [b0, b0+bs) (bs <= 64) in place, lower unit or upper, for
// right-hand side column blockIdx.x: the block goes to shared memory (coalesced), then
// a column-oriented substitution with one thread per row and one barrier per column
template <bool UPPER>
__global__ void __launch_bounds__(64) trsv_block_kernel(const double *LU, int64_t ld, double *B, int64_t ldb,
                                                        int64_t nrhs, int64_t b0, int bs) {
    __shared__ double T[64][65];
    __shared__ double x[64];
    const int64_t c = blockIdx.x;
    const int r = threadIdx.x;
    for (int e = r; e < bs * bs; e += 64) {
        const int i = e / bs, q = e - i * bs;
        T[i][q] = LU[(b0 + i) * ld + b0 + q];
    }
    double v = r < bs ? B[(b0 + r) * ldb + c] : 0.0;
    __syncthreads();
    if (!UPPER) {
        for (int q = 0; q < bs; q++) {
            if (r == q) x[q] = v;
            __syncthreads();
            if (r > q) v = fma(-T[r][q], x[q], v);
        }
    } else {
        for (int q = bs - 1; q >= 0; q--) {
            if (r == q) {
                v = v / T[q][q];
                x[q] = v;
            }
            __syncthreads();
            if (r < q) v = fma(-T[r][q], x[q], v);
        }
    }
    if (r < bs) B[(b0 + r) * ldb + c] = v;
}

// B[rows r in [r0, r1)] -= LU[r, b0:b0+bs] * B[b0:b0+bs]; warp per (row, rhs)
__global__ void trsv_update_kernel(const double *LU, int64_t ld, double *B, int64_t ldb, int64_t nrhs, int64_t b0,
                                   int bs, int64_t r0, int64_t r1) {
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int64_t rows = r1 - r0;
    if (w >= rows * nrhs) return;
    const int64_t r = r0 + w / nrhs, c = w % nrhs;
    double acc = 0.0;
    for (int q = lane; q < bs; q += 32) acc = fma(LU[r * ld + b0 + q], B[(b0 + q) * ldb + c], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) B[r * ldb + c] -= acc;
}

// ---- low precision (FP32) no-pivot LU ----------------------------------------------
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// One CTA factors the nb x nb diagonal block (nb <= 128, padded with the identity) in registers:
// 16 x 16 threads, thread (ty, tx) holding the elements (ty + 16 i, tx + 16 j), so that the
// shrinking remainder stays spread over all of them.  Two columns make a step with one barrier: the
// owners of columns and rows j, j + 1 have put their values into shared memory, every thread reads
// its eight of each and the 2 x 2 pivot block, eliminates the pair by itself and updates its
// remainder -- the next pair's columns and rows first, which go to the other buffer before the
// rest.  (One column a step: 29 us a block, the barrier and two shared-memory round trips each.)  The
// block's inverses, which only the solves read, are left to block_inverse_kernel.  One CTA per
// system of a batch: system z = blockIdx.x at A + z sA, flags at info + 2 z.
constexpr int kLuT = 16, kLuR = kNB / kLuT;  // threads per side, elements per thread and side
struct Lu128Smem {  // [buffer][column or row of the pair][thread of the other side]
    float4 c[2][2][kLuT][kLuR / 4], u[2][2][kLuT][kLuR / 4];
};
template <int JB>
__device__ __forceinline__ void put8(float4 *o, const float (&v)[kLuR]) {
    if (JB < 4) o[0] = make_float4(v[0], v[1], v[2], v[3]);
    o[1] = make_float4(v[4], v[5], v[6], v[7]);
}
template <int JB>
__device__ __forceinline__ void get8(const float4 *o, float (&v)[kLuR]) {
    if (JB < 4) {
        const float4 a = o[0];
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
    }
    const float4 b = o[1];
    v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}
template <int JB>
__device__ __forceinline__ void lu128_stage(float (&a)[kLuR][kLuR], Lu128Smem &S, int ty, int tx, int nb, int64_t k0,
                                            int *info) {
    // (the first pair of the stage; the later ones are published inside the loop)
    auto publish = [&](int jp, int b) {
        if (tx >> 1 == jp) {
            float v[kLuR];
#pragma unroll
            for (int i = 0; i < kLuR; i++) v[i] = a[i][JB];
            put8<JB>(S.c[b][tx & 1][ty], v);
        }
        if (ty >> 1 == jp) put8<JB>(S.u[b][ty & 1][tx], a[JB]);
    };
    publish(0, 0);
    __syncthreads();
#pragma unroll 1
    for (int jp = 0; jp < kLuT / 2; jp++) {
        const int buf = jp & 1, jj = 2 * jp;
        auto pivot = [&](int col, int row) { return reinterpret_cast<const float *>(S.c[buf][col][row])[JB]; };
        const float p00 = pivot(0, jj), p10 = pivot(0, jj + 1), p01 = pivot(1, jj), p11 = pivot(1, jj + 1);
        float l0[kLuR], l1[kLuR], u0[kLuR], u1[kLuR];
        get8<JB>(S.c[buf][0][ty], l0);
        get8<JB>(S.c[buf][1][ty], l1);
        get8<JB>(S.u[buf][0][tx], u0);
        get8<JB>(S.u[buf][1][tx], u1);
        const bool ok0 = p00 != 0.0f && isfinite(p00);
        const float r0 = ok0 ? rcp_approx(p00) : 0.0f, lp = p10 * r0, q11 = fmaf(-lp, p01, p11);
        const bool ok1 = q11 != 0.0f && isfinite(q11);
        const float r1 = ok1 ? rcp_approx(q11) : 0.0f;
        if (!(ok0 && ok1) && threadIdx.x == 0) {
            const int bad = JB * kLuT + jj + (ok0 ? 1 : 0);
            if (bad < nb) atomicCAS(info, 0, (int)(k0 + bad + 1));
        }
        // l0, l1: the multipliers of this thread's rows; u1: row j + 1 after row j's elimination.  Rows and
        // columns up to a pivot take no update from it.
#pragma unroll
        for (int i = JB; i < kLuR; i++) {
            l0[i] *= r0;
            l1[i] = fmaf(-l0[i], p01, l1[i]) * r1;
            u1[i] = fmaf(-lp, u0[i], u1[i]);
        }
        const float m0 = l0[JB], m1 = l1[JB];
        l0[JB] = ty > jj ? m0 : 0.0f, l1[JB] = ty > jj + 1 ? m1 : 0.0f;
        u0[JB] = tx > jj ? u0[JB] : 0.0f, u1[JB] = tx > jj + 1 ? u1[JB] : 0.0f;
#pragma unroll
        for (int i = JB; i < kLuR; i++) a[i][JB] = fmaf(-l1[i], u1[JB], fmaf(-l0[i], u0[JB], a[i][JB]));
#pragma unroll
        for (int j = JB + 1; j < kLuR; j++) a[JB][j] = fmaf(-l1[JB], u1[j], fmaf(-l0[JB], u0[j], a[JB][j]));
        if (tx >> 1 == jp) {  // the pair's own columns keep the multipliers
            const bool second = tx & 1;
#pragma unroll
            for (int i = JB; i < kLuR; i++)
                if (i > JB || ty > tx) a[i][JB] = second ? l1[i] : l0[i];
        }
        if (jp + 1 < kLuT / 2) publish(jp + 1, buf ^ 1);
#pragma unroll
        for (int i = JB + 1; i < kLuR; i++)
#pragma unroll
            for (int j = JB + 1; j < kLuR; j++) a[i][j] = fmaf(-l1[i], u1[j], fmaf(-l0[i], u0[j], a[i][j]));
        __syncthreads();
    }
    if constexpr (JB + 1 < kLuR) lu128_stage<JB + 1>(a, S, ty, tx, nb, k0, info);
}
__global__ void __launch_bounds__(kLuT *kLuT) diag_lowp_kernel(float *A, int64_t ld, int64_t k0, int nb, int *info,
                                                               int64_t sA) {
    __shared__ Lu128Smem S;
    A += blockIdx.x * sA;
    info += 2 * blockIdx.x;
    const int tx = threadIdx.x % kLuT, ty = threadIdx.x / kLuT;
    float a[kLuR][kLuR];
#pragma unroll
    for (int i = 0; i < kLuR; i++)
#pragma unroll
        for (int j = 0; j < kLuR; j++) {
            const int r = ty + kLuT * i, c = tx + kLuT * j;
            a[i][j] = r < nb && c < nb ? A[(k0 + r) * ld + k0 + c] : (r == c ? 1.0f : 0.0f);
        }
    lu128_stage<0>(a, S, ty, tx, nb, k0, info);
#pragma unroll
    for (int i = 0; i < kLuR; i++)
#pragma unroll
        for (int j = 0; j < kLuR; j++) {
            const int r = ty + kLuT * i, c = tx + kLuT * j;
            if (r < nb && c < nb) A[(k0 + r) * ld + k0 + c] = a[i][j];
        }
}

// The panels of one LU step, U12 = L11^-1 A12 and L21 = A21 U11^-1, both in one launch: a team of warps
// takes 32 NC columns (or rows) and substitutes in 32-row blocks.  Block b's right-hand side loses its
// products with the blocks before it (a warp RW of the 32 rows, lane = column), and the 32 x 32
// diagonal block's inverse, which four warps work out while the teams load their columns, is one
// more such product: no chain longer than 32.  As products with 128 x 128 inverses the panels took a
// transpose and two tensor-core launches, and the inverses as long as the diagonal block itself.
// Bound by the latency of few warps (2 per scheduler, 48 % of issue slots).  Small panels: 32 columns a
// CTA of eight warps, 4 rows each, two CTAs per SM.  Once the groups of 32 outnumber those, CTAs
// that go through several groups with the block and its inverses kept: two teams of four warps,
// 8 rows x 2 columns a lane (64 FMAs per 16 loads).  Whole factorisation at n = 9,000 (tf32) and 24,576
// (bf16), ms: 32 columns throughout 5.00, 26.5; one team of eight warps, 4 rows x 2 columns 4.92, 23.7;
// two 4.86, 23.8; two of four warps, 8 x 2 4.82, 23.7; 8 x 4 5.20, 24.2; three teams 5.03, 23.9.
constexpr int kSb = 32;
template <int NC>
struct LowpTeam {
    static constexpr int LD = 32 * NC + 1;  // row stride of the team's columns
    float H[kNB][LD];                // right-hand sides, then results: element k of column (row) i
};
template <int NC, int NT>
struct LowpPanelSmem {
    float T[kNB][kNB];               // the diagonal block's factors
    float inv[kNB / kSb][kSb][kSb];  // inverses of L's (U panel) or U's (L panel) 32 x 32 diagonal blocks
    LowpTeam<NC> team[NT];
};
// a team: 32 / RW warps of RW rows of each 32-row block
template <int RW>
constexpr int kTeamThreads = 32 * (kSb / RW);
template <int RW>
__device__ __forceinline__ void team_sync(int team) {
    asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kTeamThreads<RW>) : "memory");
}
struct LowpPanelArgs {
    float *A;
    int64_t ld, k0, nr, sA;   // trailing rows and columns k0 + 128 ... (per system)
    float *Ut;                // K-major copy of U12: column c at Ut + c ldu (null: none)
    int64_t ldu, sU;
    __nv_bfloat16 *Lb, *Ub;   // BF16 copies of L21 (row r at Lb + r ldb) and of Ut (null: none)
    int64_t ldb, sB;
    int ntu;                  // CTAs of the U panel
};
// rows [k0, k0 + nb) of the factored block, padded with the identity
template <int THREADS>
__device__ __forceinline__ void load_factors(const float *A, int64_t ld, int64_t k0, int nb, float (*T)[kNB]) {
    if (nb == kNB) {
        constexpr int Q = (kNB * kNB / 4 + THREADS - 1) / THREADS;
        float4 v[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int e = threadIdx.x + q * THREADS, r = e / (kNB / 4), c = e % (kNB / 4) * 4;
            if (e < kNB * kNB / 4) v[q] = *reinterpret_cast<const float4 *>(A + (k0 + r) * ld + k0 + c);
        }
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int e = threadIdx.x + q * THREADS;
            if (e < kNB * kNB / 4) *reinterpret_cast<float4 *>(&T[e / (kNB / 4)][e % (kNB / 4) * 4]) = v[q];
        }
    } else {
        for (int e = threadIdx.x; e < kNB * kNB; e += THREADS) {
            const int r = e / kNB, c = e % kNB;
            T[r][c] = r < nb && c < nb ? A[(k0 + r) * ld + k0 + c] : (r == c ? 1.0f : 0.0f);
        }
    }
}
// inverse of the unit-lower (or the upper) 32 x 32 block at T[b0][b0], one warp, lane = column; each
// unknown is a dot product with the ones before it, in four partial sums
template <bool LOWER>
__device__ __forceinline__ void inverse32(const float (*T)[kNB], int b0, float (*out)[kSb], int lane) {
    float x[kSb];
#pragma unroll
    for (int s = 0; s < kSb; s++) {
        const int r = LOWER ? s : kSb - 1 - s;
        float acc[4] = {r == lane ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};
        const float4 *t = reinterpret_cast<const float4 *>(&T[b0 + r][b0]);
#pragma unroll
        for (int q = 0; q < kSb / 4; q++) {
            if (LOWER ? 4 * q >= r : 4 * q + 3 <= r) continue;
            const float4 v = t[q];
            const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (LOWER ? 4 * q + e < r : 4 * q + e > r) acc[e] = fmaf(-w[e], x[4 * q + e], acc[e]);
        }
        x[r] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        if (!LOWER) x[r] *= 1.0f / T[b0 + r][b0 + r];
    }
#pragma unroll
    for (int r = 0; r < kSb; r++) out[r][lane] = x[r];
}
// acc[row][column of this lane] -= (or +=) M (RW rows from r0) . V (K rows), four of K at a time; M row-major
// from m0, or for the L panel its transpose's rows
template <bool UPANEL, int RW, int NC, int K_UNROLL, int MLD, int VLD>
__device__ __forceinline__ void panel_product(float (&acc)[RW][NC], const float *M, const float *V, int K, float sign,
                                              int lane) {
#pragma unroll K_UNROLL
    for (int k = 0; k < K; k += 4) {
        float h[4][NC];
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
            for (int c = 0; c < NC; c++) h[e][c] = sign * V[(k + e) * VLD + lane + 32 * c];
        if (UPANEL) {
#pragma unroll
            for (int i = 0; i < RW; i++) {
                const float4 t = *reinterpret_cast<const float4 *>(M + i * MLD + k);
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    acc[i][c] = fmaf(t.x, h[0][c], acc[i][c]), acc[i][c] = fmaf(t.y, h[1][c], acc[i][c]);
                    acc[i][c] = fmaf(t.z, h[2][c], acc[i][c]), acc[i][c] = fmaf(t.w, h[3][c], acc[i][c]);
                }
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
#pragma unroll
                for (int i = 0; i < RW; i += 4) {
                    const float4 t = *reinterpret_cast<const float4 *>(M + (k + e) * MLD + i);
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        acc[i][c] = fmaf(t.x, h[e][c], acc[i][c]), acc[i + 1][c] = fmaf(t.y, h[e][c], acc[i + 1][c]);
                        acc[i + 2][c] = fmaf(t.z, h[e][c], acc[i + 2][c]);
                        acc[i + 3][c] = fmaf(t.w, h[e][c], acc[i + 3][c]);
                    }
                }
        }
    }
}
// the substitution of the team's columns in its H, RW rows of each block per warp
template <bool UPANEL, int RW, int NC, int NT>
__device__ __forceinline__ void panel_solve(LowpPanelSmem<NC, NT> &S, int team, int warp, int lane) {
    constexpr int LD = LowpTeam<NC>::LD;
    LowpTeam<NC> &m = S.team[team];
    for (int b = 0; b < kNB / kSb; b++) {
        const int r0 = b * kSb + RW * warp;
        float acc[RW][NC];
#pragma unroll
        for (int i = 0; i < RW; i++)
#pragma unroll
            for (int c = 0; c < NC; c++) acc[i][c] = m.H[r0 + i][lane + 32 * c];
        panel_product<UPANEL, RW, NC, 2, kNB, LD>(acc, UPANEL ? &S.T[r0][0] : &S.T[0][r0], &m.H[0][0], b * kSb, -1.0f,
                                                  lane);
#pragma unroll
        for (int i = 0; i < RW; i++)
#pragma unroll
            for (int c = 0; c < NC; c++) m.H[r0 + i][lane + 32 * c] = acc[i][c], acc[i][c] = 0.0f;
        team_sync<RW>(team);
        panel_product<UPANEL, RW, NC, RW == 4 ? 8 : 2, kSb, LD>(
            acc, UPANEL ? &S.inv[b][RW * warp][0] : &S.inv[b][0][RW * warp], &m.H[b * kSb][0], kSb, 1.0f, lane);
        team_sync<RW>(team);  // the block's right-hand sides have been read
#pragma unroll
        for (int i = 0; i < RW; i++)
#pragma unroll
            for (int c = 0; c < NC; c++) m.H[r0 + i][lane + 32 * c] = acc[i][c];
        team_sync<RW>(team);
    }
}
// row i of the team's results (element k of column / row i), 128 contiguous values, one warp
template <int NC>
__device__ __forceinline__ float4 result4(const LowpTeam<NC> &m, int i, int lane) {
    return make_float4(m.H[4 * lane][i], m.H[4 * lane + 1][i], m.H[4 * lane + 2][i], m.H[4 * lane + 3][i]);
}
__device__ __forceinline__ void store_bf16x4(__nv_bfloat16 *o, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2 *>(o) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
}
template <int NC, int NT, int RW>
__global__ void __launch_bounds__(kTeamThreads<RW> *NT, NT == 1 ? 2 : 1) lowp_panel_kernel(LowpPanelArgs a) {
    extern __shared__ __align__(16) uint8_t raw[];
    LowpPanelSmem<NC, NT> &S = *reinterpret_cast<LowpPanelSmem<NC, NT> *>(raw);
    constexpr int CW = 32 * NC, TW = kSb / RW;  // columns and warps of a team
    constexpr int LU = 16 / NC, LL = 8;         // rows (columns of A21^T) of a warp in flight while loading
    const int team = threadIdx.x / kTeamThreads<RW>, warp = (threadIdx.x % kTeamThreads<RW>) >> 5,
              lane = threadIdx.x & 31;
    const int z = blockIdx.y;
    LowpTeam<NC> &m = S.team[team];
    float *A = a.A + z * a.sA;
    const bool up = (int)blockIdx.x < a.ntu;
    load_factors<kTeamThreads<RW> * NT>(A, a.ld, a.k0, kNB, S.T);
    __syncthreads();
    if (threadIdx.x < 32 * (kNB / kSb)) {
        const int b = threadIdx.x >> 5;
        if (up) inverse32<true>(S.T, b * kSb, S.inv[b], lane);
        else inverse32<false>(S.T, b * kSb, S.inv[b], lane);
    }
    bool first = true;
    const int64_t cta = up ? blockIdx.x : blockIdx.x - a.ntu;
    for (int64_t w0 = (cta * NT + team) * CW; first || w0 < a.nr; w0 += (int64_t)a.ntu * NT * CW) {
        const int cnt = (int)max((int64_t)0, min((int64_t)CW, a.nr - w0));
        float *A12 = A + a.k0 * a.ld + a.k0 + kNB + w0, *A21 = A + (a.k0 + kNB + w0) * a.ld + a.k0;
        if (up) {
#pragma unroll 1
            for (int q0 = warp; q0 < kNB; q0 += TW * LU) {
                float v[LU][NC];
#pragma unroll
                for (int q = 0; q < LU; q++)
#pragma unroll
                    for (int c = 0; c < NC; c++)
                        v[q][c] = lane + 32 * c < cnt ? A12[(q0 + TW * q) * a.ld + lane + 32 * c] : 0.0f;
#pragma unroll
                for (int q = 0; q < LU; q++)
#pragma unroll
                    for (int c = 0; c < NC; c++) m.H[q0 + TW * q][lane + 32 * c] = v[q][c];
            }
        } else {
            constexpr int LB = LL < CW / TW ? LL : CW / TW;
#pragma unroll 1
            for (int q0 = warp; q0 < CW; q0 += TW * LB) {
                float4 v[LB];
#pragma unroll
                for (int q = 0; q < LB; q++)
                    v[q] = q0 + TW * q < cnt ? *reinterpret_cast<const float4 *>(A21 + (q0 + TW * q) * a.ld + 4 * lane)
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int q = 0; q < LB; q++) {
                    const int i = q0 + TW * q;
                    m.H[4 * lane][i] = v[q].x, m.H[4 * lane + 1][i] = v[q].y;
                    m.H[4 * lane + 2][i] = v[q].z, m.H[4 * lane + 3][i] = v[q].w;
                }
            }
        }
        if (first) __syncthreads();  // the inverses are there, too
        else team_sync<RW>(team);
        first = false;
        if (up) panel_solve<true, RW>(S, team, warp, lane);
        else panel_solve<false, RW>(S, team, warp, lane);
        if (up) {
#pragma unroll 4
            for (int q = warp; q < kNB; q += TW)
#pragma unroll
                for (int c = 0; c < NC; c++)
                    if (lane + 32 * c < cnt) A12[q * a.ld + lane + 32 * c] = m.H[q][lane + 32 * c];
        }
#pragma unroll 2
        for (int i = warp; i < cnt; i += TW) {
            const float4 v = result4<NC>(m, i, lane);
            const int64_t r = w0 + i;
            if (!up) *reinterpret_cast<float4 *>(A21 + i * a.ld + 4 * lane) = v;
            else if (a.Ut) *reinterpret_cast<float4 *>(a.Ut + z * a.sU + r * a.ldu + 4 * lane) = v;
            if (a.Lb) store_bf16x4((up ? a.Ub : a.Lb) + z * a.sB + r * a.ldb + 4 * lane, v);
        }
        team_sync<RW>(team);  // every result is out before the next group's columns come in
    }
}
template <int NC, int NT, int RW>
static int launch_panels(LowpPanelArgs &a, int nbat, int64_t ctas, cudaStream_t st) {
    constexpr size_t smem = sizeof(LowpPanelSmem<NC, NT>);
    FLG_ONCE_PER_DEVICE(
        FLG_CUDA(cudaFuncSetAttribute(lowp_panel_kernel<NC, NT, RW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem)));
    a.ntu = (int)std::min<int64_t>(ceil_div(a.nr, 32 * NC * NT), std::max<int64_t>(1, ctas / 2 / nbat));
    lowp_panel_kernel<NC, NT, RW><<<dim3(2 * a.ntu, nbat), kTeamThreads<RW> * NT, smem, st>>>(a);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}
static int lowp_panels(LowpPanelArgs &a, int nbat, cudaStream_t st) {
    // groups of 32 columns or rows in each panel against two CTAs per SM
    const int64_t groups = ceil_div(a.nr, 32) * nbat, slots = 2LL * sm_count();
    return 2 * groups <= slots ? launch_panels<1, 1, 4>(a, nbat, slots, st)
                               : launch_panels<2, 2, 8>(a, nbat, slots / 2, st);
}

// The inverses of the diagonal blocks' unit-lower and upper factors (the solves use them), all blocks
// of all systems in one launch after the factorization: the panels' substitution applied to the
// identity.  blockIdx = (block and its 32 columns or rows, inverse of L or of U, system)
__global__ void __launch_bounds__(kTeamThreads<4>, 2) block_inverse_kernel(const float *A, int64_t ld, int64_t n, int64_t sA,
                                                                         float *Linv, float *Uinv, int64_t sD) {
    extern __shared__ __align__(16) uint8_t raw[];
    LowpPanelSmem<1, 1> &S = *reinterpret_cast<LowpPanelSmem<1, 1> *>(raw);
    LowpTeam<1> &m = S.team[0];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, w0 = (int)(blockIdx.x % 4) * 32;
    const int64_t k0 = (int64_t)(blockIdx.x / 4) * kNB;
    const bool up = blockIdx.y == 0;
    A += blockIdx.z * sA;
    float *o = (up ? Linv : Uinv) + blockIdx.z * sD + k0 * kNB;
    load_factors<kTeamThreads<4>>(A, ld, k0, (int)min((int64_t)kNB, n - k0), S.T);
    for (int k = warp; k < kNB; k += 8) m.H[k][lane] = k == w0 + lane ? 1.0f : 0.0f;
    __syncthreads();
    if (warp < kNB / kSb) {
        if (up) inverse32<true>(S.T, warp * kSb, S.inv[warp], lane);
        else inverse32<false>(S.T, warp * kSb, S.inv[warp], lane);
    }
    __syncthreads();
    if (up) {
        panel_solve<true, 4>(S, 0, warp, lane);
        for (int k = warp; k < kNB; k += 8) o[k * kNB + w0 + lane] = m.H[k][lane];
    } else {
        panel_solve<false, 4>(S, 0, warp, lane);
        for (int i = warp; i < 32; i += 8) reinterpret_cast<float4 *>(o + (w0 + i) * kNB)[lane] = result4<1>(m, i, lane);
    }
}

// C = alpha A B + beta C (row-major FP32, CUDA cores); 128x128 tiles, 8x8 per thread
constexpr int SG_BM = 128, SG_BN = 128, SG_BK = 8;
__global__ void __launch_bounds__(256) sgemm_kernel(int64_t M, int64_t N, int64_t K, float alpha, const float *A,
                                                    int64_t lda, const float *B, int64_t ldb, float beta, float *C,
                                                    int64_t ldc) {
    __shared__ float As[SG_BK][SG_BM];
    __shared__ float Bs[SG_BK][SG_BN];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int64_t row0 = (int64_t)blockIdx.y * SG_BM, col0 = (int64_t)blockIdx.x * SG_BN;
    float acc[8][8] = {};
    for (int64_t k0 = 0; k0 < K; k0 += SG_BK) {
        for (int e = threadIdx.x; e < SG_BM * SG_BK; e += 256) {
            const int r = e / SG_BK, k = e % SG_BK;
            As[k][r] = (row0 + r < M && k0 + k < K) ? A[(row0 + r) * lda + k0 + k] : 0.0f;
            const int k2 = e / SG_BN, cc = e % SG_BN;
            Bs[k2][cc] = (k0 + k2 < K && col0 + cc < N) ? B[(k0 + k2) * ldb + col0 + cc] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < SG_BK; k++) {
            float av[8], bv[8];
#pragma unroll
            for (int i = 0; i < 8; i++) av[i] = As[k][ty * 8 + i];
#pragma unroll
            for (int j = 0; j < 8; j++) bv[j] = Bs[k][tx * 8 + j];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int64_t r = row0 + ty * 8 + i;
        if (r >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int64_t c = col0 + tx * 8 + j;
            if (c < N) C[r * ldc + c] = alpha * acc[i][j] + (beta == 0.0f ? 0.0f : beta * C[r * ldc + c]);
        }
    }
}

// tensor-core update (tc_gemm.cu): C (m x nc, ldc) -= Lp (m x K, ldl) * Ut^T (nc x K, ldu), K % 128 == 0,
// for one system or a batch of them (TcBatch)
size_t tc_update_bytes(int64_t m, int64_t nc, int64_t K, int mode, int nb = 1);
int tc_update(float *C, int64_t ldc, const float *Lp, int64_t ldl, const float *Ut, int64_t ldu, int64_t m,
              int64_t nc, int64_t K, int mode, void *work, size_t work_bytes, cudaStream_t st, int *err_dev,
              int tile = 0, int max_ctas = 0, const TcBatch &bt = TcBatch{});
// the BF16 update from operands already rounded to BF16 (La, Ub: K-major __nv_bfloat16)
int tc_update_bf16(float *C, int64_t ldc, const void *La, int64_t ldl, const void *Ub, int64_t ldu, int64_t m,
                   int64_t nc, int64_t K, void *work, size_t work_bytes, cudaStream_t st, int *err_dev, int tile,
                   int max_ctas, const TcBatch &bt);

static int sgemm(cudaStream_t st, int64_t M, int64_t N, int64_t K, float alpha, const float *A, int64_t lda,
                 const float *B, int64_t ldb, float beta, float *C, int64_t ldc) {
    if (M == 0 || N == 0) return FLG_OK;
    dim3 grid((unsigned)ceil_div(N, SG_BN), (unsigned)ceil_div(M, SG_BM));
    sgemm_kernel<<<grid, 256, 0, st>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

// ---- low precision triangular solve with the diagonal-block inverses ------------------
// x = U^-1 L^-1 b for one right-hand side, FP32 factors, as a dataflow over the 128-row
// blocks in ONE cooperative launch of G CTAs.  CTA c owns the q consecutive blocks
// [c q, c q + q) (q <= kApplyQ).  In "pass order" -- the forward pass by increasing block,
// the backward pass by decreasing block -- block p needs every earlier block p' < p:
//   forward   y_i = Linv_i (b_i - sum_{j<i} L_ij y_j)
//   backward  x_i = Uinv_i (y_i - sum_{j>i} U_ij x_j).
// A CTA accumulates the contributions of the blocks before its chunk as their owners
// publish them, then runs through its own chunk locally: each finished block goes straight
// from shared memory into the later blocks of the chunk, so only one result in q crosses
// between SMs (through L2) on the critical chain.
//   * One producer thread streams the 128 x 128 FP32 slices in the order they are used
//     (for each earlier source block, its slice for every own block; for each own block,
//     its inverse, then its slices for the later own blocks) by TMA (cp.async.bulk.tensor,
//     64 KB each) into a 3-stage shared-memory ring guarded by mbarriers; rows and
//     columns outside the matrix arrive as zeros.
//   * Eight consumer warps own 16 rows of every block; lane l multiplies columns
//     4l..4l+3 of its rows (one conflict-free 16-byte load per row) by its float4 of the
//     source block and keeps 16 running partial sums per own block; finishing a block
//     reduce-scatters them over the lanes (16 shuffles).
//   * Publication is the data itself: y and x start filled with an all-ones bit pattern
//     (a NaN that FP32 arithmetic never produces; results are stored canonicalized),
//     values are stored with st.relaxed.gpu and consumers poll their four elements with
//     ld.relaxed.gpu (bounded) -- no flag, no fence.  Every wait is on a block earlier in
//     the global order (forward, then backward) and all CTAs are resident, so the order
//     always advances.
// Each block's sum runs in one CTA in a fixed order (by source block), so the result does
// not depend on G.
constexpr int kApplyConsumers = 8;                         // warps
constexpr int kApplyThreads = (kApplyConsumers + 1) * 32;  // + the producer warp
constexpr int kApplyStages = 3;
constexpr int kApplyQ = 4;                  // at most this many blocks per CTA
constexpr int kSliceBytes = kNB * kNB * 4;  // 64 KB
constexpr size_t kApplySmem = (size_t)kApplyStages * kSliceBytes + 1024;
constexpr unsigned kUnset = 0xffffffffu;

struct ApplyArgs {
    int64_t n;
    int q;           // blocks per CTA
    const float *b;  // right-hand side (FP32, n)
    float *y, *x;    // forward / backward results (n), preset to kUnset
    int *err;        // a wait ran out
};

__device__ __forceinline__ void st_relaxed_f32(float *p, float v) {
    unsigned u = __float_as_uint(v);
    if (u == kUnset) u = 0x7fffffffu;  // keep the sentinel unique
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(u) : "memory");
}
__device__ __forceinline__ void tma_load_box(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive1(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// the published float4 of a block (elements e .. e+3, those < n; zeros beyond n): the four
// loads are issued together, then those still unset are polled together until published
__device__ __forceinline__ bool fetch4(const float *v, int64_t e, int64_t n, float4 &out, int *err) {
    const int cnt = (int)max((int64_t)0, min((int64_t)4, n - e));
    unsigned u[4];
#pragma unroll
    for (int k = 0; k < 4; k++) u[k] = k < cnt ? ld_relaxed_u32(v + e + k) : 0u;
    if (!wait_published4(reinterpret_cast<const unsigned *>(v + e), cnt, kUnset, u, kWaitLimitNs, err)) return false;
    out = make_float4(__uint_as_float(u[0]), __uint_as_float(u[1]), __uint_as_float(u[2]), __uint_as_float(u[3]));
    return true;
}

// sum of acc[0..15] over the 32 lanes, scattered: lanes 2r and 2r + 1 end with row r's total
__device__ __forceinline__ float reduce_scatter16(float (&acc)[16], int lane) {
    float a8[8], a4[4], a2[2];
    const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4, h1 = lane & 2;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float send = h4 ? acc[k] : acc[8 + k];
        const float keep = h4 ? acc[8 + k] : acc[k];
        a8[k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float send = h3 ? a8[k] : a8[4 + k];
        const float keep = h3 ? a8[4 + k] : a8[k];
        a4[k] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float send = h2 ? a4[k] : a4[2 + k];
        const float keep = h2 ? a4[2 + k] : a4[k];
        a2[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
    const float send = h1 ? a2[0] : a2[1];
    const float keep = h1 ? a2[1] : a2[0];
    const float a1 = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    return a1 + __shfl_xor_sync(0xffffffffu, a1, 1);
}

// acc[sel] += S (16 rows of this warp) . v, for a run-time sel < kApplyQ
__device__ __forceinline__ void slice_fma(float (&acc)[kApplyQ][16], int sel, const float *S, float4 v) {
#pragma unroll
    for (int q = 0; q < kApplyQ; q++)
        if (q == sel) {
#pragma unroll
            for (int r = 0; r < 16; r++) {
                const float4 w = *reinterpret_cast<const float4 *>(S + r * kNB);
                acc[q][r] = fmaf(w.x, v.x, acc[q][r]);
                acc[q][r] = fmaf(w.y, v.y, acc[q][r]);
                acc[q][r] = fmaf(w.z, v.z, acc[q][r]);
                acc[q][r] = fmaf(w.w, v.w, acc[q][r]);
            }
        }
}

__global__ void __launch_bounds__(kApplyThreads, 1)
    lowp_apply_kernel(const __grid_constant__ CUtensorMap mLU, const __grid_constant__ CUtensorMap mD, ApplyArgs a) {
    extern __shared__ __align__(1024) unsigned char apply_smem[];
    float *ring = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(apply_smem) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[kApplyStages], empty[kApplyStages];
    __shared__ __align__(16) float tvec[kNB], yvec[kNB];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int nblk = (int)ceil_div(a.n, kNB);
    const int c = blockIdx.x;
    const int b0 = c * a.q, b1 = min(nblk, b0 + a.q);  // own physical blocks [b0, b1)
    const int qc = max(0, b1 - b0);
    if (t == 0) {
        for (int q = 0; q < kApplyStages; q++) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], kApplyConsumers);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (qc == 0) return;
    // pass order: forward p = i, backward p = nblk - 1 - i; own pass-order blocks [p0, p0 + qc)
    auto blk = [&](bool fwd, int p) { return fwd ? p : nblk - 1 - p; };
    if (warp == kApplyConsumers) {
        if (lane == 0) {
            long long k = 0;  // slices issued
            bool ok = true;
            auto issue = [&](const CUtensorMap *m, int x, int y) {
                const int stg = (int)(k % kApplyStages);
                if (k >= kApplyStages &&
                    !mbar_wait(&empty[stg], (uint32_t)((k / kApplyStages - 1) & 1), a.err, kWaitLimitNs)) {
                    ok = false;
                    return;
                }
                mbar_arrive_expect(&full[stg], kSliceBytes);
                tma_load_box(ring + (size_t)stg * (kNB * kNB), m, &full[stg], x, y);
                k++;
            };
            for (int pass = 0; pass < 2 && ok; pass++) {
                const bool fwd = pass == 0;
                const int p0 = fwd ? b0 : nblk - b1;
                for (int pj = 0; pj < p0 + qc && ok; pj++) {
                    const int j = blk(fwd, pj);
                    if (pj >= p0) issue(&mD, 0, (fwd ? j : nblk + j) * kNB);
                    for (int p = max(p0, pj + 1); p < p0 + qc && ok; p++) issue(&mLU, j * kNB, blk(fwd, p) * kNB);
                }
            }
            // drain: every issued load has landed before the CTA may exit
            for (long long q = k > kApplyStages ? k - kApplyStages : 0; q < k; q++)
                mbar_drain(&full[q % kApplyStages], (uint32_t)((q / kApplyStages) & 1), a.err, kWaitLimitNs);
        }
        return;
    }
    // consumers.  After a wait has run out (a.err raised, possibly by another CTA) a warp
    // keeps the loop's structure -- every stage is still waited for (each wait now returns at
    // once) and released, and every named barrier is reached -- so the producer can stop and
    // drain and no warp waits on one that has left; the results are then discarded.
    long long k = 0;  // slices consumed
    bool dead = false;
    const int row0 = warp * 16;
    auto take = [&]() -> const float * {  // the next ring stage, this warp's rows and lane's columns
        const int stg = (int)(k % kApplyStages);
        dead = !__all_sync(0xffffffffu, !dead);
        if (!mbar_wait(&full[stg], (uint32_t)((k / kApplyStages) & 1), a.err, kWaitLimitNs)) dead = true;
        return ring + (size_t)stg * (kNB * kNB) + (size_t)row0 * kNB + 4 * lane;
    };
    auto release = [&]() {
        __syncwarp();
        if (lane == 0) mbar_arrive1(&empty[k % kApplyStages]);
        k++;
    };
    for (int pass = 0; pass < 2; pass++) {
        const bool fwd = pass == 0;
        float *out_v = fwd ? a.y : a.x;  // published into and consumed from
        const int p0 = fwd ? b0 : nblk - b1;
        float acc[kApplyQ][16];
#pragma unroll
        for (int q = 0; q < kApplyQ; q++)
#pragma unroll
            for (int r = 0; r < 16; r++) acc[q][r] = 0.0f;
        // this lane's right-hand side entries of the own blocks (lanes 2r, 2r + 1 hold row r)
        float rhs[kApplyQ];
#pragma unroll
        for (int q = 0; q < kApplyQ; q++) {
            rhs[q] = 0.0f;
            if (q < qc) {
                const int64_t e = (int64_t)blk(fwd, p0 + q) * kNB + row0 + (lane >> 1);
                if (e < a.n) rhs[q] = fwd ? a.b[e] : __uint_as_float(ld_relaxed_u32(a.y + e));
            }
        }
        for (int pj = 0; pj < p0 + qc; pj++) {
            const int j = blk(fwd, pj);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (pj < p0) {
                // an earlier block, published by its owner
                if (!dead && !fetch4(out_v, (int64_t)j * kNB + 4 * lane, a.n, v, a.err)) dead = true;
            } else {
                // an own block: t = rhs - sums, then out_j = inverse . t, published and kept
                const int sel = pj - p0;
                float tmp[16];
                float rh = 0.0f;
#pragma unroll
                for (int q = 0; q < kApplyQ; q++)
                    if (q == sel) {
#pragma unroll
                        for (int r = 0; r < 16; r++) tmp[r] = acc[q][r];
                        rh = rhs[q];
                    }
                const float tot = reduce_scatter16(tmp, lane);
                if ((lane & 1) == 0) tvec[row0 + (lane >> 1)] = rh - tot;
                asm volatile("bar.sync 1, %0;" ::"r"(kApplyConsumers * 32) : "memory");
                const float4 tv = *reinterpret_cast<const float4 *>(tvec + 4 * lane);
#pragma unroll
                for (int r = 0; r < 16; r++) tmp[r] = 0.0f;
                const float *S = take();
#pragma unroll
                for (int r = 0; r < 16; r++) {
                    const float4 w = *reinterpret_cast<const float4 *>(S + r * kNB);
                    tmp[r] = fmaf(w.x, tv.x, tmp[r]);
                    tmp[r] = fmaf(w.y, tv.y, tmp[r]);
                    tmp[r] = fmaf(w.z, tv.z, tmp[r]);
                    tmp[r] = fmaf(w.w, tv.w, tmp[r]);
                }
                release();
                const float res = reduce_scatter16(tmp, lane);
                if ((lane & 1) == 0) {
                    const int r = row0 + (lane >> 1);
                    const int64_t e = (int64_t)j * kNB + r;
                    yvec[r] = e < a.n ? res : 0.0f;
                    if (e < a.n) st_relaxed_f32(out_v + e, res);
                }
                asm volatile("bar.sync 1, %0;" ::"r"(kApplyConsumers * 32) : "memory");
                v = *reinterpret_cast<const float4 *>(yvec + 4 * lane);
            }
            // (tvec and yvec are rewritten only after the next own block's first barrier, which
            // every warp reaches after its last read of them)
            for (int p = max(p0, pj + 1); p < p0 + qc; p++) {
                const float *S = take();
                slice_fma(acc, p - p0, S, v);
                release();
            }
        }
    }
}

__global__ void d2f_kernel(const double *a, float *b, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = (float)a[i];
}
// FP32 solution back to FP64; NaN everywhere if a wait of the apply ran out
__global__ void f2d_kernel(const float *a, double *b, int64_t n, const int *err) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) b[i] = *err ? __longlong_as_double(0x7ff8000000000000LL) : (double)a[i];
}

int make_box_map_f32(CUtensorMap *map, const float *base, int64_t rows, int64_t cols, int64_t ld, int box_rows,
                     int box_cols);

// blocks per CTA of the low-precision solve: 2 measured fastest on GB300 from n = 1,536 to
// 24,576 (1 hands every block between SMs; 3 and 4 lengthen each CTA's slice stream)
constexpr int kApplyQDefault = 2;

size_t lu_solve_lowp_bytes(int64_t n) {
    CountingArena c;
    c.take<float>(n);
    c.take<float>(2 * n);  // y, x: one sentinel fill
    c.take<int>(1);
    return c.bytes();
}

// the kernel attributes of the solve, set once (before any graph capture that includes it)
int lu_solve_lowp_prepare() {
    FLG_ONCE_PER_DEVICE(
        FLG_CUDA(cudaFuncSetAttribute(lowp_apply_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kApplySmem)));
    return FLG_OK;
}

int lu_solve_lowp_apply(int64_t n, const float *LU, int64_t ld, const float *dinv, const double *b, double *x,
                        void *work, size_t work_bytes, cudaStream_t st) {
    FLG_REQUIRE(ld % 4 == 0 && ((uintptr_t)LU & 15) == 0, "LU rows must be 16-byte aligned (ld % 4 == 0)");
    Arena ar(work, work_bytes);
    const int64_t nblk = ceil_div(n, kNB);
    float *bf = ar.take<float>(n);
    float *yz = ar.take<float>(2 * n);
    int *err = ar.take<int>(1);
    FLG_REQUIRE(bf && yz && err, "workspace too small for the low-precision solve");
    float *y = yz, *z = yz + n;
    // blocks per CTA: the chain crosses SMs once per q blocks; q grows only as far as the
    // CTAs' shared streams allow (one CTA per SM)
    int q = (int)std::max<int64_t>(kApplyQDefault, ceil_div(nblk, sm_count()));
    q = (int)std::min<int64_t>(q, nblk);
    FLG_REQUIRE(q <= kApplyQ, "low-precision solve: at most %lld unknowns", (long long)kApplyQ * sm_count() * kNB);
    const int G = (int)ceil_div(nblk, q);
    CUtensorMap mLU, mD;
    FLG_TRY(make_box_map_f32(&mLU, LU, n, n, ld, kNB, kNB));
    FLG_TRY(make_box_map_f32(&mD, dinv, 2 * nblk * kNB, kNB, kNB, kNB, kNB));
    d2f_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(b, bf, n);
    FLG_LAUNCH_CHECK();
    FLG_CUDA(cudaMemsetAsync(yz, 0xff, sizeof(float) * (size_t)(2 * n), st));  // the unset pattern
    FLG_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    ApplyArgs aa{n, q, bf, y, z, err};
    void *args[] = {&mLU, &mD, &aa};
    FLG_TRY(lu_solve_lowp_prepare());
    prof_begin(FLG_SLOT_LU_SOLVE, st);
    FLG_CUDA(cudaLaunchCooperativeKernel((void *)lowp_apply_kernel, dim3(G), dim3(kApplyThreads), args, kApplySmem,
                                         st));
    count_launch();
    prof_end(FLG_SLOT_LU_SOLVE, st);
    f2d_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(z, x, n, err);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

}  // namespace flg

using namespace flg;

// ---- FP64 LU entry points --------------------------------------------------------------
static int panel_geometry(int64_t m, int &nblk, int &rpc) {
    const int sms = sm_count();
    nblk = (int)std::max<int64_t>(1, std::min<int64_t>(sms, ceil_div(m, 32)));
    rpc = (int)ceil_div(m, nblk);
    return rpc <= 384 ? FLG_OK : FLG_ERR_INVALID;
}

// the identity interchanges: what the interchange kernels queued behind a panel whose wait ran out find for its columns
__global__ void identity_pivots_kernel(int32_t *ipiv, int64_t n) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) ipiv[k] = (int32_t)k;
}

// operand slices of the trailing update: L21's rows (two buffers: the next panel's slices are
// written while this panel's update still reads its own) and U12's columns, with their exponents and masks
struct SliceBufs {
    uint16_t *A[2] = {}, *B = nullptr;
    int *ea[2] = {}, *eb = nullptr;
    SliceMask *ma[2] = {}, *mb = nullptr;
    template <class Ar>
    void carve(Ar &ar, int64_t n) {
        const size_t rows = n > kPanel ? (size_t)n : 0;
        for (int k = 0; k < 2; k++) {
            A[k] = ar.template take<uint16_t>(kSlices * rows * kSliceK);
            ea[k] = ar.template take<int>(rows);
            ma[k] = ar.template take<SliceMask>(rows);
        }
        B = ar.template take<uint16_t>(kSlices * rows * kSliceK);
        eb = ar.template take<int>(rows);
        mb = ar.template take<SliceMask>(rows);
    }
};

extern "C" size_t flg_lu_factor_f64_workspace(int64_t n) {
    CountingArena c;
    const int nblk = sm_count();
    c.take<GridBar>(1);
    c.take<unsigned long long>(2 * nblk);
    c.take<double>((size_t)2 * nblk * kRowBufLd);
    c.take<double>(2 * kPanel);
    SliceBufs sb;
    sb.carve(c, n);
    return c.bytes();
}

// Per host thread and device: the streams of the FP64 LU's look-ahead -- the next panel
// (highest priority) beside the trailing update, and the interchanges of the columns left of
// each panel (lowest priority), which nothing reads until the factorization ends.
struct F64Streams {
    int dev = -1;
    cudaStream_t panel = nullptr, left = nullptr;
    cudaEvent_t next_ready = nullptr, panel_done = nullptr, panel_on = nullptr, factored = nullptr, left_done = nullptr;
};
constexpr int kF64StreamDevices = 64;
static int f64_streams(F64Streams **out) {
    thread_local F64Streams per_dev[kF64StreamDevices];
    int dev = 0;
    FLG_CUDA(cudaGetDevice(&dev));
    FLG_REQUIRE(dev >= 0 && dev < kF64StreamDevices, "device ordinal %d out of range", dev);
    F64Streams &fs = per_dev[dev];
    if (fs.dev != dev) {
        int lo = 0, hi = 0;
        FLG_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
        FLG_CUDA(cudaStreamCreateWithPriority(&fs.panel, cudaStreamNonBlocking, hi));
        FLG_CUDA(cudaStreamCreateWithPriority(&fs.left, cudaStreamNonBlocking, lo));
        for (cudaEvent_t *e : {&fs.next_ready, &fs.panel_done, &fs.panel_on, &fs.factored, &fs.left_done})
            FLG_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
        fs.dev = dev;
    }
    *out = &fs;
    return FLG_OK;
}

extern "C" int flg_lu_factor_f64(int64_t n, double *A, int64_t ld, int32_t *ipiv, int *info, void *work,
                                 size_t work_bytes, void *stream) {
    FLG_RANGE("flg_lu_factor_f64");
    FLG_REQUIRE(n >= 0 && ld >= n && info, "bad LU arguments");
    *info = 0;
    if (n == 0) return FLG_OK;
    FLG_REQUIRE(A && ipiv, "null pointer");
    int nblk0, rpc0;
    FLG_REQUIRE(panel_geometry(n, nblk0, rpc0) == FLG_OK, "FP64 dense LU supports n <= %d (use GMRES above)",
                sm_count() * 384);
    cudaStream_t st = as_stream(stream);
    Arena ar(work, work_bytes);
    const int maxblk = sm_count(), near = slice_near_range(n);
    GridBar *bar = ar.take<GridBar>(1);
    unsigned long long *word = ar.take<unsigned long long>(2 * maxblk);
    double *rowbuf = ar.take<double>((size_t)2 * maxblk * kRowBufLd);
    double *diagbuf = ar.take<double>(2 * kPanel);
    SliceBufs sb;
    sb.carve(ar, n);
    FLG_REQUIRE(diagbuf != nullptr && (n <= kPanel || sb.mb != nullptr), "workspace too small for LU (%zu bytes)",
                work_bytes);
    F64Streams *fs = nullptr;
    FLG_TRY(f64_streams(&fs));
    FLG_ONCE_PER_DEVICE(
        FLG_CUDA(cudaFuncSetAttribute(panel_f64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      384 * kPanel * (int)sizeof(double))));
    FLG_CUDA(cudaMemsetAsync(bar, 0, sizeof(GridBar), st));
    if (n > kClusterPanelRows) {
        identity_pivots_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(ipiv, n);
        FLG_LAUNCH_CHECK();
    }
    // the panel of columns [k0, k0 + kb), rows k0.. on stream s, and the slices of its L21;
    // started (optional) completes once the panel's first kernel is resident
    auto panel = [&](int64_t k0, cudaStream_t s, cudaEvent_t started) -> int {
        const int kb = (int)std::min<int64_t>(kPanel, n - k0);
        const int64_t m = n - k0;
        const int b = (int)(k0 / kPanel) & 1;
        if (m <= kClusterPanelRows) {
            // two halves on a cluster, the second updated by the first in between
            const int h0 = std::min(kHalf, kb), h1 = kb - h0;
            prof_begin(FLG_SLOT_LU_PANEL, s);
            FLG_TRY(cluster_panel({A, ld, n, k0, h0, ipiv, &bar->info, &bar->err, (int)k0 + h0,
                                   (int)k0 + kb, 1, 0},
                                  started, s));
            if (h1 > 0) {
                FLG_TRY(half_update(A, ld, k0 + kHalf, n, k0, h1, s));
                FLG_TRY(cluster_panel({A, ld, n, k0 + kHalf, h1, ipiv, &bar->info, &bar->err, (int)k0,
                                       (int)k0 + kHalf, 0, 0},
                                      nullptr, s));
            }
            prof_end(FLG_SLOT_LU_PANEL, s);
            return slice_rows(A + (k0 + kb) * ld + k0, ld, m - kb, n, sb.A[b], sb.ea[b], sb.ma[b], near, s);
        }
        int nblk, rpc;
        panel_geometry(m, nblk, rpc);
        int per_sm = 0;
        const size_t smem = (size_t)rpc * kb * sizeof(double);
        FLG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, panel_f64_kernel, 256, smem));
        FLG_REQUIRE(per_sm * sm_count() >= nblk, "panel grid (%d CTAs) cannot be co-resident", nblk);
        // both buffers of the published words to parity 1 (columns 0 and 1 expect parity 0)
        FLG_CUDA(cudaMemsetAsync(word, 0x80, 2 * (size_t)maxblk * sizeof(unsigned long long), s));
        PanelArgs pa{A, ld, n, k0, kb, rpc, ipiv, bar, word, rowbuf, diagbuf};
        void *args[] = {&pa};
        prof_begin(FLG_SLOT_LU_PANEL, s);
        FLG_CUDA(cudaLaunchCooperativeKernel((void *)panel_f64_kernel, dim3(nblk), dim3(256), args, smem, s));
        count_launch();
        prof_end(FLG_SLOT_LU_PANEL, s);
        return slice_rows(A + (k0 + kb) * ld + k0, ld, m - kb, n, sb.A[b], sb.ea[b], sb.ma[b], near, s);
    };
    // Look-ahead: after each panel's trailing update has reached the next panel's 64 columns,
    // the next panel factors on the panel stream while the main stream updates the rest.
    // The interchanges of the columns left of each panel go to the left stream, in order.
    FLG_CUDA(cudaEventRecord(fs->factored, st));
    FLG_CUDA(cudaStreamWaitEvent(fs->left, fs->factored, 0));  // the left stream starts after prior work
    FLG_TRY(panel(0, st, nullptr));
    bool ahead = false;  // the current panel ran ahead on the panel stream
    for (int64_t k0 = 0; k0 < n; k0 += kPanel) {
        const int kb = (int)std::min<int64_t>(kPanel, n - k0);
        if (ahead) FLG_CUDA(cudaStreamWaitEvent(st, fs->panel_done, 0));
        if (k0 > 0) {
            FLG_CUDA(cudaEventRecord(fs->factored, st));
            FLG_CUDA(cudaStreamWaitEvent(fs->left, fs->factored, 0));
            swap_rows_kernel<<<(unsigned)ceil_div(k0, kSwapCols), kSwapThreads, 0, fs->left>>>(A, ld, ipiv, k0, kb,
                                                                                                   0, k0);
            FLG_LAUNCH_CHECK();
        }
        const int64_t c0 = k0 + kb;
        ahead = false;
        if (c0 >= n) break;
        const int64_t nc = n - c0;
        const int64_t nn = std::min<int64_t>(kPanel, nc);  // the next panel's columns first
        // where the substitution of all columns is a long launch (37 us from 2,432 columns on, 12 for the next
        // panel's), the rest of them follows beside the panel; at fewer columns the launch costs what it saves.
        // Factorizations in ms without this / at any width: 2,432 5.96 / 6.02, 2,800 7.27 / 7.24, 3,200 8.77 / 8.58, 3,600
        // 10.39 / 9.98, 4,608 14.68 / 14.11, 7,000 31.25 / 31.17
        const bool split = nc >= kTrsmWide * (int64_t)sm_count() && nc <= kClusterPanelRows;
        FLG_TRY(swap_trsm(A, ld, ipiv, k0, c0, split ? c0 + nn : n, sb.B, n, sb.eb, sb.mb, near, st));
        prof_begin(FLG_SLOT_LU_UPDATE, st);
        const int b = (int)(k0 / kPanel) & 1;
        const double *L21 = A + c0 * ld + k0, *U12 = A + k0 * ld + c0;
        FLG_TRY(slice_update(A + c0 * ld + c0, ld, nc, nn, L21, U12, sb.A[b], n, sb.ea[b], sb.ma[b], sb.B, n, 0, sb.eb,
                             sb.mb, near, &bar->err, maxblk, st));
        if (nc > nn) {
            FLG_CUDA(cudaEventRecord(fs->next_ready, st));
            FLG_CUDA(cudaStreamWaitEvent(fs->panel, fs->next_ready, 0));
            // a cluster panel keeps its SMs out of the update's persistent grid, which waits until
            // the cluster is resident (16 SMs of one GPC are never free at once under that grid)
            const bool cluster = nc <= kClusterPanelRows;
            FLG_TRY(panel(c0, fs->panel, cluster ? fs->panel_on : nullptr));
            FLG_CUDA(cudaEventRecord(fs->panel_done, fs->panel));
            ahead = true;
            if (cluster) FLG_CUDA(cudaStreamWaitEvent(st, fs->panel_on, 0));
            if (split) FLG_TRY(swap_trsm(A, ld, ipiv, k0, c0 + nn, n, sb.B + nn * kSliceK, n, sb.eb + nn, sb.mb + nn, near, st));
            FLG_TRY(slice_update(A + c0 * ld + c0 + nn, ld, nc, nc - nn, L21, U12 + nn, sb.A[b], n, sb.ea[b], sb.ma[b],
                                 sb.B, n, nn, sb.eb, sb.mb, near, &bar->err, cluster ? maxblk - kPanelCtas : maxblk, st));
        }
        prof_end(FLG_SLOT_LU_UPDATE, st);
        if (!ahead) FLG_TRY(panel(c0, st, nullptr));  // the last panel: nothing to overlap it with
    }
    FLG_CUDA(cudaEventRecord(fs->left_done, fs->left));
    FLG_CUDA(cudaStreamWaitEvent(st, fs->left_done, 0));
    GridBar hb;
    FLG_CUDA(cudaMemcpyAsync(&hb, bar, sizeof(GridBar), cudaMemcpyDeviceToHost, st));
    FLG_CUDA(cudaStreamSynchronize(st));
    if (hb.err) {
        set_error("a bounded device wait timed out (LU panel exchange or tensor-core update)");
        return FLG_ERR_TIMEOUT;
    }
    *info = hb.info;
    if (hb.info) {
        set_error("Matrix is singular (zero pivot at row %d)", hb.info - 1);
        return FLG_ERR_SINGULAR;
    }
    return FLG_OK;
}

// A solve takes one cluster of 16 SMs per right-hand side, so few right-hand sides run at once
// (six fit GB300); the two launches per 64 rows below spread all right-hand sides over the SMs.  Measured,
// ms cluster / launches: n = 684: 1: 0.19 / 0.58, 16: 0.55 / 0.66, 32: 0.91 / 0.73;
// n = 4,608: 1: 1.25 / 4.67, 32: 6.2 / 9.6, 64: 13.7 / 14.6.
static bool solve_on_cluster(int64_t n, int64_t nrhs) { return nrhs <= (n >= 2048 ? 32 : 16) && trsv_fits(n); }

// err (optional): a device word that a timed-out wait of the solve raises
static int lu_solve_f64(int64_t n, int64_t nrhs, const double *LU, int64_t ld, const int32_t *ipiv, double *B, int64_t ldb,
                        int *err, cudaStream_t st) {
    if (solve_on_cluster(n, nrhs)) return trsv_cluster(n, nrhs, LU, ld, ipiv, B, ldb, err, st);
    if (n <= kPivSmemMax) {
        FLG_ONCE_PER_DEVICE(
            FLG_CUDA(cudaFuncSetAttribute(apply_pivots_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          kPivSmemMax * (int)sizeof(double))));
        apply_pivots_smem_kernel<<<(unsigned)nrhs, 256, n * sizeof(double), st>>>(B, ldb, ipiv, n);
    } else {
        apply_pivots_kernel<<<(unsigned)ceil_div(nrhs, 32), 32, 0, st>>>(B, ldb, nrhs, ipiv, n);
    }
    FLG_LAUNCH_CHECK();
    const int bsz = 64;
    for (int64_t b0 = 0; b0 < n; b0 += bsz) {
        const int bs = (int)std::min<int64_t>(bsz, n - b0);
        trsv_block_kernel<false><<<(unsigned)nrhs, 64, 0, st>>>(LU, ld, B, ldb, nrhs, b0, bs);
        FLG_LAUNCH_CHECK();
        if (b0 + bs < n) {
            const int64_t rows = n - b0 - bs;
            trsv_update_kernel<<<(unsigned)ceil_div(rows * nrhs * 32, 256), 256, 0, st>>>(LU, ld, B, ldb, nrhs, b0,
                                                                                         bs, b0 + bs, n);
            FLG_LAUNCH_CHECK();
        }
    }
    for (int64_t b0 = ((n - 1) / bsz) * bsz; b0 >= 0; b0 -= bsz) {
        const int bs = (int)std::min<int64_t>(bsz, n - b0);
        trsv_block_kernel<true><<<(unsigned)nrhs, 64, 0, st>>>(LU, ld, B, ldb, nrhs, b0, bs);
        FLG_LAUNCH_CHECK();
        if (b0 > 0) {
            trsv_update_kernel<<<(unsigned)ceil_div(b0 * nrhs * 32, 256), 256, 0, st>>>(LU, ld, B, ldb, nrhs, b0, bs,
                                                                                       0, b0);
            FLG_LAUNCH_CHECK();
        }
    }
    return FLG_OK;
}

static int check_solve(int64_t n, int64_t nrhs, int64_t ld, int64_t ldb) {
    FLG_REQUIRE(n >= 0 && nrhs >= 0 && ld >= n && ldb >= nrhs, "bad LU solve arguments");
    FLG_REQUIRE(nrhs <= 65535 || n == 0, "at most 65,535 right-hand sides per call");
    return FLG_OK;
}
extern "C" int flg_lu_solve_f64(int64_t n, int64_t nrhs, const double *LU, int64_t ld, const int32_t *ipiv, double *B,
                                int64_t ldb, void *stream) {
    FLG_RANGE("flg_lu_solve_f64");
    FLG_TRY(check_solve(n, nrhs, ld, ldb));
    if (n == 0 || nrhs == 0) return FLG_OK;
    return lu_solve_f64(n, nrhs, LU, ld, ipiv, B, ldb, nullptr, as_stream(stream));
}
extern "C" int flg_lu_solve_f64_flag(int64_t n, int64_t nrhs, const double *LU, int64_t ld, const int32_t *ipiv, double *B,
                                     int64_t ldb, int *flag, void *stream) {
    FLG_RANGE("flg_lu_solve_f64_flag");
    FLG_TRY(check_solve(n, nrhs, ld, ldb));
    FLG_REQUIRE(flag != nullptr, "null flag");
    FLG_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), as_stream(stream)));
    if (n == 0 || nrhs == 0) return FLG_OK;
    return lu_solve_f64(n, nrhs, LU, ld, ipiv, B, ldb, flag, as_stream(stream));
}

// ---- low-precision LU entry points ----------------------------------------------------
// Per host thread and device: the stream that runs the next diagonal block while the
// trailing update finishes (highest priority), and the events of that fork and join.
// Created on first use; an LU captured in a graph makes one eager pass first.
// One set per device ordinal, so a thread that moves between GPUs keeps (and reuses) each
// device's stream and events instead of creating new ones on every switch.
struct SideStream {
    int dev = -1;
    cudaStream_t s = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
constexpr int kSideStreamDevices = 64;
static int side_stream(SideStream **out) {
    thread_local SideStream per_dev[kSideStreamDevices];
    int dev = 0;
    FLG_CUDA(cudaGetDevice(&dev));
    FLG_REQUIRE(dev >= 0 && dev < kSideStreamDevices, "device ordinal %d out of range", dev);
    SideStream &ss = per_dev[dev];
    if (ss.dev != dev) {
        int lo = 0, hi = 0;
        FLG_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
        FLG_CUDA(cudaStreamCreateWithPriority(&ss.s, cudaStreamNonBlocking, hi));
        FLG_CUDA(cudaEventCreateWithFlags(&ss.fork, cudaEventDisableTiming));
        FLG_CUDA(cudaEventCreateWithFlags(&ss.join, cudaEventDisableTiming));
        ss.dev = dev;
    }
    *out = &ss;
    return FLG_OK;
}

extern "C" int64_t flg_lu_lowp_dinv_elems(int64_t n) { return 2 * ceil_div(std::max<int64_t>(n, 1), kNB) * kNB * kNB; }

// Tensor-core modes defer most of the trailing update, on two levels: blocks are grouped into middle
// panels of W1 columns [K1, E) and those into outer panels of W columns [K0, E2).  Inner step k0
// (diagonal block, panels) updates only the L-shaped part of the Schur complement that the next
// inner steps read -- rows > k0 x columns (k0, E), and rows (k0, E) x columns >= E -- with
// rank-128 updates; after a middle panel the rest of the outer panel's columns and rows get one
// rank-W1 update, and rows and columns >= E2 one rank-W update per outer panel.  A tile of C
// costs the update kernel 1.9 GB of traffic per 472 million elements whatever the depth (rank 1,024 at
// 15,360: 268 us of products alone, 358 us of C alone, 464 us together), so a deeper rank moves the trailing
// matrix less often.  The K-major copy of U (UtB: one row of W per column >= K0) feeds all three.
// Measured, factor with copies: W1 = W = 512 / W1 = W = 1,024 / 512 and 1,024 / 512 and 2,048:
// n = 9,000 tf32 4.96 / 4.87 / 4.87 / 4.93 ms, bf16 4.58 / 4.44 / 4.40 / 4.43; n = 24,576 tf32
// 34.2 / 32.0 / 31.2 / 31.7, bf16 30.4 / 25.5 / 24.4 / 23.5 (bf16 products take half as long, so that
// C's traffic weighs more).  Below 8,192 unknowns one level of 512 is the fastest (4,608: 1.99, two
// levels 2.05).
static int64_t inner_width() { return 4 * (int64_t)kNB; }
static int64_t outer_width(int64_t n, int mode) {
    return inner_width() * (n < 8192 ? 1 : mode == FLG_LU_BF16 ? 4 : 2);
}

// scratch of nbat systems, system z's at + z n W floats; BF16 mode: the BF16 copies of the outer
// panel's L columns and of UtB (n W each per system) in PB
template <class Ar>
static void lowp_carve(Ar &ar, int64_t n, int nbat, int mode, float **UtB, char **tcw, size_t *tcb,
                       __nv_bfloat16 **PB) {
    const int64_t W = outer_width(n, mode);
    *UtB = ar.template take<float>((size_t)nbat * n * W);
    // the updates take their operands as they are (TF32, or PB's BF16 copies): no operand workspace
    *tcb = (mode == FLG_LU_FP32) ? 0 : tc_update_bytes(n, n, W, FLG_LU_TF32, nbat);
    *tcw = ar.template take<char>(*tcb);
    *PB = mode == FLG_LU_BF16 ? ar.template take<__nv_bfloat16>((size_t)2 * nbat * n * W) : nullptr;
}

// precision part of an LU mode (the tile bits masked off)
static int lu_prec(int mode) { return mode & ~(FLG_LU_TILE_N128 | FLG_LU_TILE_N256); }

extern "C" size_t flg_lu_factor_lowp_workspace(int64_t n, int mode) {
    mode = lu_prec(mode);
    CountingArena c;
    float *d;
    char *w;
    size_t t;
    __nv_bfloat16 *pb;
    lowp_carve(c, n, 1, mode, &d, &w, &t, &pb);
    return c.bytes() + 256;  // + the flags of flg_lu_factor_lowp, at the end
}

extern "C" size_t flg_lu_factor_lowp_batched_workspace(int64_t n, int nbat, int mode) {
    mode = lu_prec(mode);
    CountingArena c;
    float *d;
    char *w;
    size_t t;
    __nv_bfloat16 *pb;
    lowp_carve(c, n, std::max(nbat, 1), mode, &d, &w, &t, &pb);
    return c.bytes();
}

// The low-precision LU of nbat systems of order n in one sequence of launches: system z at
// A + z sA (row stride ld), its block inverses at dinv + z flg_lu_lowp_dinv_elems(n), its
// flags at flags + 2 z.  Every kernel of a step covers all systems (one CTA per system for
// the diagonal blocks; the tensor-core updates walk the tiles of all systems).
static int lowp_factor(int64_t n, int nbat, float *A, int64_t ld, int64_t sA, int mode, float *dinv, int *flags,
                       void *work, size_t work_bytes, cudaStream_t st) {
    FLG_REQUIRE(n >= 0 && ld >= n && flags && nbat >= 1, "bad LU arguments");
    const int tbits = mode & (FLG_LU_TILE_N128 | FLG_LU_TILE_N256);
    FLG_REQUIRE(tbits != (FLG_LU_TILE_N128 | FLG_LU_TILE_N256), "two tile widths in LU mode %d", mode);
    const int tile = tbits == FLG_LU_TILE_N128 ? 128 : tbits == FLG_LU_TILE_N256 ? 256 : 0;
    mode = lu_prec(mode);
    FLG_REQUIRE(mode == FLG_LU_TF32 || mode == FLG_LU_BF16 || (mode == FLG_LU_FP32 && tile == 0), "unknown LU mode %d",
                mode | tbits);
    FLG_REQUIRE(nbat == 1 || mode != FLG_LU_FP32, "batched LU needs a tensor-core mode (TF32 or BF16)");
    FLG_REQUIRE(nbat == 1 || (sA >= n * ld && sA % 4 == 0), "bad system stride");
    FLG_REQUIRE(ld % 4 == 0, "ld must be a multiple of 4 (16-byte rows)");
    FLG_CUDA(cudaMemsetAsync(flags, 0, 2 * sizeof(int) * nbat, st));
    if (n == 0) return FLG_OK;
    FLG_REQUIRE(A && dinv, "null pointer");
    Arena ar(work, work_bytes);
    float *UtB;
    char *tcw;
    size_t tcb;
    __nv_bfloat16 *PB;
    lowp_carve(ar, n, nbat, mode, &UtB, &tcw, &tcb, &PB);
    FLG_REQUIRE(UtB && (tcb == 0 || tcw) && (mode != FLG_LU_BF16 || PB), "workspace too small for LU (%zu bytes)",
                work_bytes);
    int *dinfo = flags;  // [0] first bad pivot, [1] tensor-core wait timed out
    const int64_t W = outer_width(n, mode), W1 = inner_width();  // outer and middle panel width
    // per-system strides: the matrix, the block inverses, U's K-major copy
    const int64_t sD = flg_lu_lowp_dinv_elems(n), sUt = n * W;
    const TcBatch bA{nbat, sA, sA, sUt};
    // BF16 mode: each step's finished L and U panels are rounded once into LB (row r, column
    // c - K0 of the outer panel at LB + r W + c - K0) and UB (laid out as UtB), and every
    // trailing update of the outer panel reads them
    __nv_bfloat16 *LB = PB, *UB = PB ? PB + (size_t)nbat * n * W : nullptr;
    const TcBatch bB{nbat, sA, n * W, n * W};
    int64_t K0 = 0;  // first column of the current outer panel
    // C -= Lp Up^T (Lp inside A at columns [K0, E), Up inside UtB) over m x nc, depth K
    auto upd = [&](float *C, const float *Lp, const float *Up, int64_t m, int64_t nc, int64_t K, int ctas) -> int {
        if (mode == FLG_LU_BF16) {
            const int64_t off = Lp - A, r = off / ld, c = off % ld;
            return tc_update_bf16(C, ld, LB + r * W + (c - K0), W, UB + (Up - UtB), W, m, nc, K, tcw, tcb, st,
                                  dinfo + 1, tile, ctas, bB);
        }
        return tc_update(C, ld, Lp, ld, Up, W, m, nc, K, mode, tcw, tcb, st, dinfo + 1, tile, ctas, bA);
    };
    FLG_ONCE_PER_DEVICE(
        FLG_CUDA(cudaFuncSetAttribute(block_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(LowpPanelSmem<1, 1>))));
    const bool tc = mode != FLG_LU_FP32;
    const int64_t nblk = ceil_div(n, kNB);
    SideStream *side = nullptr;
    if (tc) FLG_TRY(side_stream(&side));
    // the persistent updates that run beside the look-ahead diagonal blocks leave them an SM each
    const int cap = std::max(1, sm_count() - nbat);
    auto diag = [&](int64_t d0, cudaStream_t s) {
        prof_begin(FLG_SLOT_LU_DIAG, s);
        diag_lowp_kernel<<<nbat, kLuT * kLuT, 0, s>>>(A, ld, d0, (int)std::min<int64_t>(kNB, n - d0), dinfo, sA);
        prof_end(FLG_SLOT_LU_DIAG, s);
    };
    // Look-ahead: once the 128 x 128 block at d0 has its last update (launched on st), the
    // diagonal kernel of that block runs on the side stream while st goes on with the rest of
    // the trailing update; the next panels wait for it.
    bool pending = false;
    auto look_ahead = [&](int64_t d0) -> int {
        FLG_CUDA(cudaEventRecord(side->fork, st));
        FLG_CUDA(cudaStreamWaitEvent(side->s, side->fork, 0));
        diag(d0, side->s);
        FLG_LAUNCH_CHECK();
        FLG_CUDA(cudaEventRecord(side->join, side->s));
        pending = true;
        return FLG_OK;
    };
    // C[r0:, c0:] -= L U^T over columns [ka, kb) for rows [r0, r1) and columns [c0, c1): the first
    // diagonal block of it, at (r0, c0), first when `ahead`, so that it factors beside the rest
    auto block = [&](int64_t r0, int64_t r1, int64_t c0, int64_t c1, int64_t ka, int64_t kb, bool ahead) -> int {
        float *C = A + r0 * ld + c0, *Lp = A + r0 * ld + ka, *Up = UtB + (c0 - K0) * W + (ka - K0);
        const int64_t m = r1 - r0, nc = c1 - c0, K = kb - ka;
        if (!ahead || m <= kNB) return upd(C, Lp, Up, m, nc, K, pending ? cap : 0);
        FLG_TRY(upd(C, Lp, Up, std::min<int64_t>(kNB, m), std::min<int64_t>(kNB, nc), K, 0));
        FLG_TRY(look_ahead(r0));
        FLG_TRY(upd(C + kNB * ld, Lp + kNB * ld, Up, m - kNB, std::min<int64_t>(kNB, nc), K, cap));
        if (nc > kNB) FLG_TRY(upd(C + kNB, Lp, Up + kNB * W, m, nc - kNB, K, cap));
        return FLG_OK;
    };
    for (K0 = 0; K0 < n; K0 += W) {
        const int64_t E2 = std::min<int64_t>(n, K0 + W);
        for (int64_t K1 = K0; K1 < E2; K1 += W1) {
            const int64_t E = std::min<int64_t>(n, K1 + W1);
            for (int64_t k0 = K1; k0 < E; k0 += kNB) {
                const int nb = (int)std::min<int64_t>(kNB, n - k0);
                if (pending) {  // this block's diagonal kernel ran ahead on the side stream
                    FLG_CUDA(cudaStreamWaitEvent(st, side->join, 0));
                    pending = false;
                } else {
                    diag(k0, st);
                    FLG_LAUNCH_CHECK();
                }
                const int64_t c0 = k0 + nb, nr = n - c0;
                if (nr <= 0) continue;
                prof_begin(FLG_SLOT_LU_PANEL, st);
                // (nb < kNB only for the last block, which has no trailing part)
                float *A12 = A + k0 * ld + c0, *A21 = A + c0 * ld + k0;
                float *Ut = UtB + (c0 - K0) * W + (k0 - K0);  // row: column - K0; K offset: k0 - K0
                LowpPanelArgs pa{A, ld, k0, nr, sA, tc ? Ut : nullptr, W, sUt, nullptr, nullptr, W, n * W, 0};
                if (mode == FLG_LU_BF16) pa.Ut = nullptr, pa.Lb = LB + c0 * W + (k0 - K0), pa.Ub = UB + (Ut - UtB);
                FLG_TRY(lowp_panels(pa, nbat, st));
                prof_end(FLG_SLOT_LU_PANEL, st);
                prof_begin(FLG_SLOT_LU_UPDATE, st);
                if (!tc) {
                    FLG_TRY(sgemm(st, nr, nr, nb, -1.0f, A21, ld, A12, ld, 1.0f, A + c0 * ld + c0, ld));
                } else if (E > c0) {
                    FLG_TRY(block(c0, n, c0, E, k0, c0, true));         // rows > k0 x columns (k0, E)
                    if (n > E) FLG_TRY(block(c0, E, E, n, k0, c0, false));  // rows (k0, E) x columns >= E
                }
                prof_end(FLG_SLOT_LU_UPDATE, st);
            }
            if (tc && E2 > E) {  // the middle panel's rank-W1 update of the rest of the outer panel
                prof_begin(FLG_SLOT_LU_UPDATE, st);
                FLG_TRY(block(E, n, E, E2, K1, E, true));
                if (n > E2) FLG_TRY(block(E, E2, E2, n, K1, E, false));
                prof_end(FLG_SLOT_LU_UPDATE, st);
            }
        }
        if (tc && n > E2) {  // the deferred rank-W update of rows and columns >= E2
            prof_begin(FLG_SLOT_LU_UPDATE, st);
            FLG_TRY(block(E2, n, E2, n, K0, E2, true));
            prof_end(FLG_SLOT_LU_UPDATE, st);
        }
    }
    if (pending) FLG_CUDA(cudaStreamWaitEvent(st, side->join, 0));  // (every look-ahead is joined above)
    block_inverse_kernel<<<dim3((unsigned)(4 * nblk), 2, nbat), kTeamThreads<4>, sizeof(LowpPanelSmem<1, 1>), st>>>(
        A, ld, n, sA, dinv, dinv + nblk * kNB * kNB, sD);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

extern "C" int flg_lu_factor_lowp_async(int64_t n, float *A, int64_t ld, int mode, float *dinv, int *flags, void *work,
                                        size_t work_bytes, void *stream) {
    FLG_RANGE("flg_lu_factor_lowp_async");
    return lowp_factor(n, 1, A, ld, 0, mode, dinv, flags, work, work_bytes, as_stream(stream));
}

extern "C" int flg_lu_factor_lowp_batched_async(int64_t n, int nbat, float *A, int64_t ld, int64_t stride_a, int mode,
                                                float *dinv, int *flags, void *work, size_t work_bytes,
                                                void *stream) {
    FLG_RANGE("flg_lu_factor_lowp_batched_async");
    FLG_REQUIRE(nbat >= 1 && nbat <= 64, "batch of %d systems (1 .. 64)", nbat);
    return lowp_factor(n, nbat, A, ld, stride_a, mode, dinv, flags, work, work_bytes, as_stream(stream));
}

extern "C" int flg_lu_factor_lowp(int64_t n, float *A, int64_t ld, int mode, float *dinv, int *info, void *work,
                                  size_t work_bytes, void *stream) {
    FLG_RANGE("flg_lu_factor_lowp");
    FLG_REQUIRE(info, "null info");
    *info = 0;
    FLG_REQUIRE(n >= 0 && ld >= n, "bad LU arguments");
    if (n == 0) return FLG_OK;
    // the two device flags live at the end of the workspace
    const size_t need = flg_lu_factor_lowp_workspace(n, mode);
    FLG_REQUIRE(work && work_bytes >= need, "workspace too small for LU (%zu bytes, %zu needed)", work_bytes, need);
    int *flags = (int *)((char *)work + ((need - 64) & ~size_t(15)));
    cudaStream_t st = as_stream(stream);
    FLG_TRY(flg_lu_factor_lowp_async(n, A, ld, mode, dinv, flags, work, need - 128, stream));
    int hflags[2] = {0, 0};
    FLG_CUDA(cudaMemcpyAsync(hflags, flags, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    FLG_CUDA(cudaStreamSynchronize(st));
    if (hflags[1]) {
        set_error("a bounded device wait timed out (tensor-core update)");
        return FLG_ERR_TIMEOUT;
    }
    *info = hflags[0];
    if (hflags[0]) {
        set_error("zero or non-finite pivot at row %d in the low-precision LU", hflags[0] - 1);
        return FLG_ERR_SINGULAR;
    }
    return FLG_OK;
}

extern "C" size_t flg_lu_solve_lowp_workspace(int64_t n) { return lu_solve_lowp_bytes(n); }

extern "C" int flg_lu_solve_lowp(int64_t n, const float *LU, int64_t ld, const float *dinv, const double *b, double *x,
                                 void *work, size_t work_bytes, void *stream) {
    FLG_RANGE("flg_lu_solve_lowp");
    FLG_REQUIRE(n >= 0 && ld >= n, "bad solve arguments");
    if (n == 0) return FLG_OK;
    return lu_solve_lowp_apply(n, LU, ld, dinv, b, x, work, work_bytes, as_stream(stream));
}
