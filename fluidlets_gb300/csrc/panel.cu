// panel.cu -- partial-pivoting LU of a narrow FP64 panel on one thread-block cluster.
//
// The m x kb panel (kb <= 32, m <= kClusterPanelRows) of the FP64 LU (lu.cu) with LAPACK getf2's
// pivot choice (the largest |a| of the column, the first row on ties).  What limits a panel is
// the exchange of pivot candidates once per column.  Through L2 between all SMs a round costs
// about 4 us (a released flag, a poll, and then the pivot row); here one cluster of up to 16
// CTAs holds the whole panel, one thread per row, and a round is a few remote shared-memory
// stores and one hardware cluster barrier.
//
// CTA c owns rows k0 + c rpc ..., all kb columns of them in shared memory (Pm): finished multipliers
// left of the current column, right of it the values as of the last full update.  Column j:
//   1. warp w < W, rows 32 w ..: the interchange of column j - 1 on its rows, their multipliers, and
//      column j's values; the warp's largest |x| (two 32-bit reductions over the bits, which order
//      like the value; NaN never wins) and a copy of that row, and of row k0 + j;
//   2. publisher warps: eight pick the CTA's candidate, complete its row (one FMA per lane) and
//      send it to every CTA of the cluster, one sends the candidate's key, local row and
//      reciprocal, two send row k0 + j like the eight;
//   3. the row warps, beside the exchange: the rest of the rank-1 update of column j - 1;
//   4. every row warp picks the winner among the CTAs' candidates (ties: the smaller CTA, which
//      owns the smaller rows).
// The exchange is st.async: the data's arrival completes the receiver's mbarrier, so a round has
// no acknowledgement (measured with 16 CTAs: 490-700 clocks; plain remote stores and a cluster
// barrier 1,215; bulk copies 1,700).  Received rows are buffered three deep: a CTA sends column
// j + 3's after it has column j + 2's from every CTA, and those leave after every use of column j's.
// FP64 is what a column costs otherwise: GB300 issues one FP64 warp instruction per 64 clocks and
// scheduler whatever its active lanes (comparisons and reciprocals included), so tests run on
// integer bits, the reciprocal is three FMAs on the 20-bit approximation, and a panel of few rows
// gives each row several warps (groups of columns) for the rank-1 update so that all four
// schedulers have some.
// Every element gets the same FMAs in the same column order as in the textbook loop, so factors
// and pivots do not depend on the cluster size or the grouping.
//
// After the panel: its interchanges on a few companion columns (the other half of a 64-column
// block), and with `trsm` also U12 = L11^-1 A12 on them, one warp per column.
#include <algorithm>

#include "cluster.cuh"
#include "flg_common.cuh"
#include "panel.cuh"
#include "waits.cuh"

namespace flg {

constexpr int kRowPubs = 8, kKeyPub = kRowPubs, kDiagPubs = 2;
constexpr int kPubWarps = kRowPubs + 1 + kDiagPubs, kMaxRowWarps = 16;
constexpr int kPmLd = kHalf + 1;
constexpr int kRx = 3;  // buffers of received candidates

struct PanelShared {
    double rx_row[kRx][kPanelCtas][kHalf];
    double rx_diag[kRx][kHalf];  // row k0 + j
    double rx_rcp[kRx][kPanelCtas];
    unsigned long long rx_key[kRx][kPanelCtas];
    unsigned long long rx_lrow[kRx][kPanelCtas];
    // candidates of this CTA, by column parity: a publisher may still read column j's while the row
    // warps copy column j + 1's
    double stage[2][kMaxRowWarps][kHalf], dstage[2][kHalf];
    unsigned long long skey[2][kMaxRowWarps];
    int srow[2][kMaxRowWarps];
    int swin[2];  // the last column's winner (-1: none), for the publishers
    int piv[kHalf], dst[2 * kHalf], src[2 * kHalf];
    double L11[kHalf][kPmLd];
    unsigned long long bar[kRx];
};

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

__global__ void __launch_bounds__(32 * (kMaxRowWarps + kPubWarps), 1) panel_cluster_kernel(ClusterPanelArgs a) {
    extern __shared__ __align__(16) uint8_t raw[];
    PanelShared &S = *reinterpret_cast<PanelShared *>(raw);
    double *Pm = reinterpret_cast<double *>(raw + ((sizeof(PanelShared) + 15) & ~size_t(15)));  // [32 W][kPmLd]
    const int c = blockIdx.x, ncta = gridDim.x, kb = a.kb, rpc = a.rpc;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, rw = (int)(blockDim.x >> 5) - kPubWarps;
    const int pub = warp - rw;                 // publisher warp, or negative: a row warp
    const int W = (rpc + 31) >> 5, CG = rw / W;  // row blocks of 32, column groups of the rank-1 update
    const int rb = warp % W, cg = warp / W;    // row warps: row block, column group
    const int k0 = (int)a.k0, r0 = k0 + c * rpc;
    const int nr = max(0, min(rpc, (int)a.n - r0));
    if (t == 0) {
        for (int b = 0; b < kRx; b++) mbar_init((uint64_t *)&S.bar[b], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int l0 = warp; l0 < nr; l0 += 8 * (int)(blockDim.x >> 5)) {
        double v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int lr = l0 + k * (int)(blockDim.x >> 5);
            v[k] = lr < nr && lane < kb ? a.A[(int64_t)(r0 + lr) * a.ld + k0 + lane] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int lr = l0 + k * (int)(blockDim.x >> 5);
            if (lr < nr) Pm[lr * kPmLd + lane] = v[k];
        }
    }
    __syncthreads();
    const int lr = rb * 32 + lane, row = r0 + lr;  // row warps: this lane's row
    double *mine = Pm + (size_t)lr * kPmLd;        // (inside the allocation for every lane of a row warp)
    const bool have = pub < 0 && lr < nr;
    cluster_sync();  // every CTA's mbarriers are ready

    // what a CTA receives per column: a row, a key, a row index and a reciprocal from each CTA, and row k0 + j
    const uint32_t rx_bytes = (uint32_t)ncta * (8 * kHalf + 24) + 8 * kHalf;
    int buf = 0, pbuf = 0, prow = -1;
    uint32_t parity = 0;
    const double *pv = nullptr;  // the previous column's pivot row, by column
    double rcp = 0.0;
    bool ok = false;
    for (int j = 0; j < kb; j++) {
        const int g = k0 + j;
        double l = 0.0;
        if (pub < 0 && cg == 0) {
            if (j > 0) {  // column j - 1's interchange on this warp's rows (finished rows included)
                const int gl = g - 1 - r0, pl = prow - r0;
                if (prow != g - 1 && pl >= 0 && pl < nr && (pl >> 5) == rb) Pm[pl * kPmLd + lane] = S.rx_diag[pbuf][lane];
                if (gl >= 0 && gl < nr && (gl >> 5) == rb) Pm[gl * kPmLd + lane] = pv[lane];
                __syncwarp();
            }
            double v = mine[j];
            if (j > 0) {
                l = mine[j - 1];
                if (ok) {
                    l *= rcp;
                    v = fma(-l, pv[j], v);
                }
                if (have && row >= g) mine[j - 1] = l, mine[j] = v;
            }
            const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
            const unsigned long long key = have && row >= g && b <= 0x7ff0000000000000ull ? b + 1ull : 0ull;
            const int w = warp_argmax(key);
            __syncwarp();
            // whole rows: multipliers, column j, and columns j + 1 ... without column j - 1's update
            if (w >= 0) S.stage[j & 1][rb][lane] = Pm[(rb * 32 + w) * kPmLd + lane];
            if ((g - r0) >> 5 == rb && g - r0 < nr) S.dstage[j & 1][lane] = Pm[(g - r0) * kPmLd + lane];
            if (lane == (w < 0 ? 0 : w)) {
                S.skey[j & 1][rb] = key;
                S.srow[j & 1][rb] = lr;
            }
        }
        __syncthreads();
        if (pub >= 0) {
            const void *bar = &S.bar[buf];
            if (j > 0) {
                const int win = S.swin[(j - 1) & 1];
                pv = win >= 0 ? S.rx_row[pbuf][win] : S.rx_diag[pbuf];
                ok = finite_nonzero(pv[j - 1]);
            }
            if (pub <= kKeyPub) {
                if (pub == kKeyPub && lane == 0) expect_tx(bar, rx_bytes);
                const unsigned long long key = lane < W ? S.skey[j & 1][lane] : 0ull;
                const int w = warp_argmax(key);
                const double *st = S.stage[j & 1][w < 0 ? 0 : w];
                if (pub == kKeyPub) {
                    const double p = w >= 0 ? st[j] : 0.0;
                    const double rp = finite_nonzero(p) ? fast_rcp(p) : 0.0;
                    if (lane < ncta) {
                        send(&S.rx_key[buf][c], bar, lane, w >= 0 ? S.skey[j & 1][w] : 0ull);
                        send(&S.rx_lrow[buf][c], bar, lane, (unsigned long long)(w >= 0 ? S.srow[j & 1][w] : 0));
                        send(&S.rx_rcp[buf][c], bar, lane, rp);
                    }
                } else {
                    double y = st[lane];
                    if (j > 0 && ok && lane > j) y = fma(-st[j - 1], pv[lane], y);
                    for (int d = pub; d < ncta; d += kRowPubs) send(&S.rx_row[buf][c][lane], bar, d, y);
                }
            } else if (g >= r0 && g < r0 + nr) {
                const double *st = S.dstage[j & 1];
                double y = st[lane];
                if (j > 0 && ok && lane > j) y = fma(-st[j - 1], pv[lane], y);
                for (int d = pub - kKeyPub - 1; d < ncta; d += kDiagPubs) send(&S.rx_diag[buf][lane], bar, d, y);
            }
            pbuf = buf;
            if (++buf == kRx) buf = 0;
            continue;
        }
        if (j > 0 && ok) {  // the rest of the previous column's rank-1 update, beside the exchange
            if (cg > 0) l = mine[j - 1];
            for (int q0 = j + 1 + cg; q0 < kb; q0 += 4 * CG) {
                double y[4], u[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int q = min(q0 + k * CG, kHalf - 1);
                    y[k] = mine[q];
                    u[k] = pv[q];
                }
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (q0 + k * CG < kb) {
                        const double z = fma(-l, u[k], y[k]);
                        if (row >= g) mine[q0 + k * CG] = z;
                    }
            }
        }
        if (CG > 1) asm volatile("bar.sync 1, %0;" ::"r"(32 * rw) : "memory");  // the other groups' columns of this row
        cluster_wait((uint64_t *)&S.bar[buf], parity, a.err, kWaitLimitNs);
        __syncwarp();
        const int win = warp_argmax(lane < ncta ? S.rx_key[buf][lane] : 0ull);
        // no candidate anywhere (a column of NaN): row g stays, as the pivot
        pv = win >= 0 ? S.rx_row[buf][win] : S.rx_diag[buf];
        rcp = win >= 0 ? S.rx_rcp[buf][win] : 0.0;
        ok = finite_nonzero(pv[j]);
        prow = win >= 0 ? k0 + win * rpc + (int)S.rx_lrow[buf][win] : g;
        prow = min(max(prow, g), (int)a.n - 1);  // (in range also after a wait that ran out: it indexes memory)
        if (warp == 0 && lane == 0) {
            S.swin[j & 1] = win;
            S.piv[j] = prow;
            if (c == 0) a.ipiv[g] = prow;
            if (c == 0 && !ok) atomicCAS(a.info, 0, g + 1);
        }
        pbuf = buf;
        if (++buf == kRx) buf = 0, parity ^= 1;
    }
    if (pub < 0 && cg == 0) {  // the last column's interchange and multipliers
        const int gl = k0 + kb - 1 - r0, pl = prow - r0;
        if (prow != k0 + kb - 1 && pl >= 0 && pl < nr && (pl >> 5) == rb) Pm[pl * kPmLd + lane] = S.rx_diag[pbuf][lane];
        if (gl >= 0 && gl < nr && (gl >> 5) == rb) Pm[gl * kPmLd + lane] = pv[lane];
        __syncwarp();
        if (have && row >= k0 + kb && ok) mine[kb - 1] *= rcp;
    }
    __syncthreads();
    for (int l0 = warp; l0 < nr; l0 += blockDim.x >> 5)
        if (lane < kb) a.A[(int64_t)(r0 + l0) * a.ld + k0 + lane] = Pm[l0 * kPmLd + lane];
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
    FLG_ONCE_PER_DEVICE(
        FLG_CUDA(cudaFuncSetAttribute(panel_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        FLG_CUDA(cudaFuncSetAttribute(panel_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)panel_smem(32 * kMaxRowWarps))));
    int ncta = 1;
    while (ncta < kPanelCtas && (int64_t)ncta * 32 < m) ncta *= 2;
    a.rpc = (int)ceil_div(m, ncta);
    const int W = (int)ceil_div(a.rpc, 32), CG = std::max(1, 8 / W);  // eight row warps where the rows fill fewer
    const int threads = (W * CG + kPubWarps) * 32;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ncta);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = panel_smem(32 * W);
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
    FLG_CUDA(cudaLaunchKernelEx(&cfg, panel_cluster_kernel, a));
    count_launch();
    return FLG_OK;
}

}  // namespace flg
