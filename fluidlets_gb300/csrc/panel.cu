// panel.cu -- partial-pivoting LU of a narrow FP64 panel on one thread-block cluster.
//
// The m x kb panel (kb <= 32, m <= kClusterPanelRows) of the FP64 LU (lu.cu) with LAPACK getf2's
// pivot choice (the largest |a| of the column, the first row on ties).  What limits a panel is
// the exchange of pivot candidates once per column.  Through L2 between all SMs a round costs
// about 4 us (a released flag, a poll, and then the pivot row); here one cluster of up to 16
// CTAs holds the whole panel, one thread per row, and a round is a few remote shared-memory
// stores and one hardware cluster barrier.
//
// Thread lr of CTA c owns row k0 + c rpc + lr: the columns from the current one on live in its
// registers, moved down by one with every column (the rank-1 update writes a[i - 1] from a[i]), the
// finished multipliers in shared memory (Pm).  Column j:
//   1. rows below pivot j - 1: multiplier, and column j's value; each warp's largest |x| (two
//      32-bit reductions over the bits, which order like the value; NaN never wins), whose thread
//      stages its remaining row;
//   2. publisher warps, beside the row warps: four pick the CTA's candidate, complete its row
//      (one FMA per lane) and send it to every CTA of the cluster, one sends the candidate's key
//      and reciprocal, two do the same as the four for row k0 + j;
//   3. the rest of the rank-1 update of column j - 1, beside the exchange;
//   4. every warp picks the winner among the CTAs' candidates (ties: the smaller CTA, which owns
//      the smaller rows); the winner's thread takes over row k0 + j, which the pivot row replaces.
// The exchange is st.async: the data's arrival completes the receiver's mbarrier, so a round has
// no acknowledgement (measured with 16 CTAs: 490 clocks; plain remote stores and a cluster
// barrier 1,215).  Received rows are buffered three deep: a CTA sends column j + 3's after it has
// column j + 2's from every CTA, and those leave after every use of column j's.
// FP64 is what a column costs otherwise: GB300 issues one FP64 warp instruction per 64 clocks and
// scheduler whatever its active lanes (comparisons and reciprocals included), so tests run on
// integer bits and the reciprocal is three FMAs on the 20-bit approximation.
// Every element gets the same FMAs in the same column order as in the textbook loop, so factors
// and pivots do not depend on the cluster size.
//
// After the panel: its interchanges on a few companion columns (the other half of a 64-column
// block), and with `trsm` also U12 = L11^-1 A12 on them, one warp per column.
#include <algorithm>

#include "flg_common.cuh"
#include "panel.cuh"
#include "waits.cuh"

namespace flg {

constexpr int kRowPubs = 4, kKeyPub = kRowPubs, kDiagPubs = 2;
constexpr int kPubWarps = kRowPubs + 1 + kDiagPubs, kMaxRowWarps = 12;
constexpr int kPmLd = kHalf + 1;
constexpr int kRx = 3;  // buffers of received candidates

struct PanelShared {
    double rx_row[kRx][kPanelCtas][kHalf];
    double rx_diag[kRx][2 * kHalf];  // row k0 + j; the upper half stays unused padding for shifted reads
    double rx_rcp[kRx][kPanelCtas];
    unsigned long long rx_key[kRx][kPanelCtas];
    unsigned long long rx_lrow[kRx][kPanelCtas];
    // candidates of this CTA, by column parity: a publisher may still read column j's while the row
    // warps stage column j + 1's
    double2 stage[2][kMaxRowWarps][kHalf / 2], dstage[2][kHalf / 2];
    unsigned long long skey[2][kMaxRowWarps];
    int srow[2][kMaxRowWarps];
    int piv[kHalf], dst[2 * kHalf], src[2 * kHalf];
    double L11[kHalf][kPmLd];
    unsigned long long bar[kRx];
};

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

__device__ __forceinline__ bool finite_nonzero(double p) {  // on the bits: FP64 comparisons are slow
    const unsigned long long u = (unsigned long long)__double_as_longlong(p) << 1;
    return u != 0 && u < 0xffe0000000000000ull;
}
// 1 / p to the last bit or two: the third-order iteration r (1 + e + e^2), e = 1 - p r, from the
// 20-bit approximation; scaled to stay clear of denormals
__device__ __forceinline__ double fast_rcp(double p) {
    const int ex = (__double2hiint(p) >> 20) & 0x7ff;
    if (ex < 64 || ex > 1982) return __drcp_rn(p);
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(p));
    const double e = fma(-p, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// the lane with the largest key, the lowest one on ties; -1 if every key is 0
__device__ __forceinline__ int warp_argmax(unsigned long long key) {
    const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
    const unsigned h = __reduce_max_sync(0xffffffffu, hi);
    const unsigned l = __reduce_max_sync(0xffffffffu, hi == h ? lo : 0u);
    const unsigned who = __ballot_sync(0xffffffffu, hi == h && lo == l);
    return (h | l) ? __ffs(who) - 1 : -1;
}

// MAXW: the most row warps of a launch; 9 (4,608 rows) leaves 128 registers per thread, 12 only 96
template <int MAXW>
__global__ void __launch_bounds__(32 * (MAXW + kPubWarps), 1) panel_cluster_kernel(ClusterPanelArgs a) {
    extern __shared__ __align__(16) uint8_t raw[];
    PanelShared &S = *reinterpret_cast<PanelShared *>(raw);
    double *Pm = reinterpret_cast<double *>(raw + ((sizeof(PanelShared) + 15) & ~size_t(15)));  // [rpc][kPmLd]
    const int c = blockIdx.x, ncta = gridDim.x, kb = a.kb, rpc = a.rpc;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, rw = (int)(blockDim.x >> 5) - kPubWarps;
    const int pub = warp - rw;  // publisher warp, or negative: a row warp
    const int k0 = (int)a.k0, r0 = k0 + c * rpc;
    const int nr = max(0, min(rpc, (int)a.n - r0));
    if (t == 0) {
        for (int b = 0; b < kRx; b++) mbar_init((uint64_t *)&S.bar[b], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int lr = warp; lr < nr; lr += blockDim.x >> 5)
        if (lane < kb) Pm[lr * kPmLd + lane] = a.A[(int64_t)(r0 + lr) * a.ld + k0 + lane];
    __syncthreads();
    const int row = r0 + t;  // row warps only
    const bool have = pub < 0 && t < nr;
    double x[kHalf];  // columns j, j + 1, ... of this thread's row
#pragma unroll
    for (int i = 0; i < kHalf; i++) x[i] = have && i < kb ? Pm[t * kPmLd + i] : 0.0;
    cluster_sync();  // every CTA's mbarriers are ready

    // what a CTA receives per column: a row, a key, a row index and a reciprocal from each CTA, and row k0 + j
    const uint32_t rx_bytes = (uint32_t)ncta * (8 * kHalf + 24) + 8 * kHalf;
    const double *pv = nullptr;  // the previous column's pivot row, by column
    double rcp = 0.0;
    bool ok = false;
    int buf = 0;
    uint32_t parity = 0;
    for (int j = 0; j < kb; j++) {
        const int g = k0 + j;
        double l = 0.0, v = x[0];
        if (pub < 0) {
            if (j > 0) {
                l = ok ? x[0] * rcp : x[0];
                v = ok ? fma(-l, pv[j], x[1]) : x[1];
                if (have && row >= g) Pm[t * kPmLd + j - 1] = l;
            }
            const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
            const unsigned long long key = have && row >= g && b <= 0x7ff0000000000000ull ? b + 1ull : 0ull;
            const int w = warp_argmax(key);
            const bool diag = have && row == g;
            if (lane == w || diag) {  // columns j, j + 1, ..., of which all but j lack column j - 1's update
                double2 *st = lane == w ? S.stage[j & 1][warp] : S.dstage[j & 1];
#pragma unroll
                for (int i = 0; i < kHalf; i += 2)
                    if (j + i < kb) {
                        const double2 p = j > 0 ? make_double2(i ? x[i + 1 < kHalf ? i + 1 : kHalf - 1] : v,
                                                               x[i + 2 < kHalf ? i + 2 : kHalf - 1])
                                                : make_double2(x[i], x[i + 1]);
                        st[i / 2] = p;
                        if (diag) S.dstage[j & 1][i / 2] = p;
                    }
            }
            if (lane == (w < 0 ? 0 : w)) {
                S.skey[j & 1][warp] = key;
                S.srow[j & 1][warp] = t;
            }
        }
        __syncthreads();
        if (pub >= 0) {
            const void *bar = &S.bar[buf];
            if (pub == kKeyPub && lane == 0) expect_tx(&S.bar[buf], rx_bytes);
            if (pub <= kKeyPub) {
                const int w = warp_argmax(lane < rw ? S.skey[j & 1][lane] : 0ull);
                const int lr = w >= 0 ? S.srow[j & 1][w] : 0;
                const double *st = reinterpret_cast<const double *>(S.stage[j & 1][w < 0 ? 0 : w]);
                if (pub == kKeyPub) {
                    if (lane < ncta) {
                        send(&S.rx_key[buf][c], bar, lane, w >= 0 ? S.skey[j & 1][w] : 0ull);
                        send(&S.rx_lrow[buf][c], bar, lane, (unsigned long long)lr);
                    }
                    const double p = w >= 0 ? st[0] : 0.0;
                    const double rp = finite_nonzero(p) ? fast_rcp(p) : 0.0;
                    if (lane < ncta) send(&S.rx_rcp[buf][c], bar, lane, rp);
                } else {
                    double y = lane < j ? Pm[lr * kPmLd + lane] : st[lane - j];
                    if (j > 0 && ok && lane > j) y = fma(-Pm[lr * kPmLd + j - 1], pv[lane], y);
                    for (int d = pub; d < ncta; d += kRowPubs) send(&S.rx_row[buf][c][lane], bar, d, y);
                }
            } else if (g >= r0 && g < r0 + nr) {
                const int lr = g - r0;
                double y = lane < j ? Pm[lr * kPmLd + lane] : reinterpret_cast<const double *>(S.dstage[j & 1])[lane - j];
                if (j > 0 && ok && lane > j) y = fma(-Pm[lr * kPmLd + j - 1], pv[lane], y);
                for (int d = pub - kKeyPub - 1; d < ncta; d += kDiagPubs) send(&S.rx_diag[buf][lane], bar, d, y);
            }
            // no publisher still reads Pm when the pivot row and row g change places below
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kPubWarps) : "memory");
        } else if (j > 0) {  // the rest of the previous column's rank-1 update, beside the exchange
            x[0] = v;
            if (ok) {
#pragma unroll
                for (int ib = 0; ib < kHalf; ib += 4)
                    if (j + ib < kb)
#pragma unroll
                        for (int i = ib; i < ib + 4; i++)
                            if (i >= 1) x[i] = fma(-l, pv[min(j + i, kHalf - 1)], x[i + 1 < kHalf ? i + 1 : kHalf - 1]);
            } else {
#pragma unroll
                for (int i = 1; i + 1 < kHalf; i++) x[i] = x[i + 1];
            }
        }
        cluster_wait((uint64_t *)&S.bar[buf], parity, a.err);
        __syncwarp();
        const int win = warp_argmax(lane < ncta ? S.rx_key[buf][lane] : 0ull);
        // no candidate anywhere (a column of NaN): row g stays, as the pivot
        pv = win >= 0 ? S.rx_row[buf][win] : S.rx_diag[buf];
        rcp = win >= 0 ? S.rx_rcp[buf][win] : 0.0;
        ok = finite_nonzero(pv[j]);
        const int prow = win >= 0 ? k0 + win * rpc + (int)S.rx_lrow[buf][win] : g;
        if (pub < 0) {
            if (have && row == prow && prow != g) {  // the old row g moves here
#pragma unroll
                for (int i = 0; i < kHalf; i++) x[i] = S.rx_diag[buf][j + i];
            }
        } else if (pub == kKeyPub) {
            const int pl = prow - r0, gl = g - r0;
            if (pl >= 0 && pl < nr && prow != g && lane < j) Pm[pl * kPmLd + lane] = S.rx_diag[buf][lane];
            if (gl >= 0 && gl < nr && lane < kb) Pm[gl * kPmLd + lane] = pv[lane];
            if (lane == 0) {
                S.piv[j] = prow;
                if (c == 0) a.ipiv[g] = prow;
                if (c == 0 && !ok) atomicCAS(a.info, 0, g + 1);
            }
        }
        if (++buf == kRx) buf = 0, parity ^= 1;
    }
    if (have && row >= k0 + kb) Pm[t * kPmLd + kb - 1] = ok ? x[0] * rcp : x[0];
    __syncthreads();
    for (int lr = warp; lr < nr; lr += blockDim.x >> 5)
        if (lane < kb) a.A[(int64_t)(r0 + lr) * a.ld + k0 + lane] = Pm[lr * kPmLd + lane];
    // the panel's interchanges on the companion columns [cc0, cc1): slots as in lu.cu
    for (int s = t; s < 2 * kHalf; s += blockDim.x) {
        const int q = s & (kHalf - 1);
        int r = q < kb ? k0 + q : -1;
        if (s >= kHalf && q < kb) {
            r = S.piv[q] >= k0 + kb ? S.piv[q] : -1;
            for (int p = 0; p < q; p++) r = S.piv[p] == r ? -1 : r;
        }
        S.dst[s] = r;
        for (int p = kb - 1; p >= 0; p--) {
            const int f = k0 + p, b = S.piv[p];
            r = r == f ? b : r == b ? f : r;
        }
        S.src[s] = r;
    }
    cluster_sync();
    if (a.trsm) {
        for (int e = t; e < kb * kb; e += blockDim.x)
            S.L11[e / kb][e % kb] = __ldcg(a.A + (int64_t)(k0 + e / kb) * a.ld + k0 + e % kb);
    }
    __syncthreads();
    for (int cc = a.cc0 + c + ncta * warp; cc < a.cc1; cc += ncta * (int)(blockDim.x >> 5)) {
        const int d0 = S.dst[lane], d1 = S.dst[kHalf + lane];
        double y = d0 >= 0 ? a.A[(int64_t)S.src[lane] * a.ld + cc] : 0.0;
        const double z = d1 >= 0 ? a.A[(int64_t)S.src[kHalf + lane] * a.ld + cc] : 0.0;
        __syncwarp();
        if (d1 >= 0) a.A[(int64_t)d1 * a.ld + cc] = z;
        if (a.trsm)
            for (int q = 0; q + 1 < kb; q++) {
                const double yq = __shfl_sync(0xffffffffu, y, q);
                if (lane > q && lane < kb) y = fma(-S.L11[lane][q], yq, y);
            }
        if (d0 >= 0) a.A[(int64_t)d0 * a.ld + cc] = y;
    }
}

// C (m x nc, nc <= 32) -= L (m x 32) U (32 x nc), all in A: the second half of a 64-column block
// updated by its first half before that half's panel runs.  A warp per two rows, lane = column, the
// FMAs of an element in the textbook's order: 64 FP64 instructions of 64 clocks per warp, so a
// small panel takes 2 us and a tall one fills the FP64 pipes of every SM (4,608 rows: 9 us).
constexpr int kHalfRows = 2, kHalfWarps = 4;
__global__ void __launch_bounds__(32 * kHalfWarps) half_update_kernel(double *A, int64_t ld, int64_t r0, int64_t n,
                                                                      int64_t k0, int nc) {
    __shared__ double U[kHalf][kHalf], L[kHalfWarps][kHalfRows][kHalf];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t rb = r0 + ((int64_t)blockIdx.x * kHalfWarps + warp) * kHalfRows;
    double u[kHalf / kHalfWarps], acc[kHalfRows];
#pragma unroll
    for (int k = 0; k < kHalf / kHalfWarps; k++)
        u[k] = lane < nc ? A[(k0 + warp + k * kHalfWarps) * ld + k0 + kHalf + lane] : 0.0;
#pragma unroll
    for (int i = 0; i < kHalfRows; i++) {
        const bool in = rb + i < n;
        L[warp][i][lane] = in ? A[(rb + i) * ld + k0 + lane] : 0.0;
        acc[i] = in && lane < nc ? A[(rb + i) * ld + k0 + kHalf + lane] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kHalf / kHalfWarps; k++) U[warp + k * kHalfWarps][lane] = u[k];
    __syncthreads();
    if (lane >= nc) return;
#pragma unroll
    for (int k = 0; k < kHalf; k++)
#pragma unroll
        for (int i = 0; i < kHalfRows; i++) acc[i] = fma(-L[warp][i][k], U[k][lane], acc[i]);
#pragma unroll
    for (int i = 0; i < kHalfRows; i++)
        if (rb + i < n) A[(rb + i) * ld + k0 + kHalf + lane] = acc[i];
}

int half_update(double *A, int64_t ld, int64_t r0, int64_t n, int64_t k0, int nc, cudaStream_t st) {
    if (r0 >= n || nc <= 0) return FLG_OK;
    half_update_kernel<<<(unsigned)ceil_div(n - r0, kHalfRows * kHalfWarps), 32 * kHalfWarps, 0, st>>>(A, ld, r0, n, k0,
                                                                                                    nc);
    FLG_LAUNCH_CHECK();
    return FLG_OK;
}

static size_t panel_smem(int rpc) { return ((sizeof(PanelShared) + 15) & ~size_t(15)) + sizeof(double) * rpc * kPmLd; }

// The panel of columns [k0, k0 + kb) on stream st; started (optional): an event that completes
// once the cluster is resident, so that a grid that would fill the device can wait for it.
int cluster_panel(const ClusterPanelArgs &in, cudaEvent_t started, cudaStream_t st) {
    ClusterPanelArgs a = in;
    const int64_t m = a.n - a.k0;
    FLG_REQUIRE(a.kb >= 1 && a.kb <= kHalf && m <= kClusterPanelRows, "bad cluster panel");
    static bool attr_set = false;
    if (!attr_set) {
        for (const void *k : {(const void *)panel_cluster_kernel<9>, (const void *)panel_cluster_kernel<kMaxRowWarps>}) {
            FLG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            FLG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)panel_smem(32 * kMaxRowWarps)));
        }
        attr_set = true;
    }
    int ncta = 1;
    while (ncta < kPanelCtas && (int64_t)ncta * 32 < m) ncta *= 2;
    a.rpc = (int)ceil_div(m, ncta);
    const int threads = (int)(ceil_div(a.rpc, 32) + kPubWarps) * 32;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ncta);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = panel_smem(a.rpc);
    cfg.stream = st;
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ncta;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
    if (started) {
        at[1].id = cudaLaunchAttributeLaunchCompletionEvent;
        at[1].val.launchCompletionEvent.event = started;
        at[1].val.launchCompletionEvent.flags = 0;
        cfg.numAttrs = 2;
    }
    cfg.attrs = at;
    FLG_CUDA(cudaLaunchKernelEx(&cfg, a.rpc <= 9 * 32 ? panel_cluster_kernel<9> : panel_cluster_kernel<kMaxRowWarps>, a));
    count_launch();
    return FLG_OK;
}

}  // namespace flg
