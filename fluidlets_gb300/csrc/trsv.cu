// trsv.cu -- the triangular solves of the FP64 LU for few right-hand sides, one launch.
//
// x = U^-1 L^-1 P b.  One cluster of 16 CTAs per right-hand side; 32-row blocks are dealt to the CTAs
// in turn.  A block's owner accumulates the products with the earlier blocks' results as they
// arrive (forward: blocks 0, 1, ..., backward: last to first), solves its 32 x 32 diagonal block and
// sends the 32 values into every CTA's shared memory (st.async, completing the receiver's
// mbarrier of that block), so a solve is one dependency chain of block solves with a few hundred clocks of
// exchange instead of two launches per 64 rows.  Per block on the chain: the product with the
// previous block (32 x 32 FMAs on four warps, 8 FP64 instructions of 64 clocks each), four
// partial sums, and the substitution (32 steps of a shuffle and an FMA); everything else -- products with earlier blocks,
// matrix loads, the interchanges -- runs ahead of it.
// Measured on GB300, n = 4,608, one right-hand side: see flg_lu_solve_f64 (lu.cu).
#include <algorithm>

#include "cluster.cuh"
#include "flg_common.cuh"
#include "trsv.cuh"

namespace flg {

constexpr int kTb = 32, kTvCtas = 16, kTvWarps = 8, kTvThreads = 32 * kTvWarps;
constexpr int kSwapBlock = 64;  // interchanges composed at a time

struct TrsvShared {
    double T[kTb][kTb + 1];        // the diagonal block
    double ps[kTvWarps][kTb], pl[4][kTb];  // partial sums: earlier blocks, the previous block
    double out[kTb];
    int piv[kTvWarps][kSwapBlock], dst[kTvWarps][2 * kSwapBlock], src[kTvWarps][2 * kSwapBlock];
    int err;
};

__global__ void __launch_bounds__(kTvThreads, 1) trsv_cluster_kernel(const double *LU, int64_t ld, const int32_t *ipiv,
                                                                     double *B, int64_t ldb, int n, int *err) {
    extern __shared__ __align__(16) uint8_t raw[];
    TrsvShared &S = *reinterpret_cast<TrsvShared *>(raw);
    const int nb = (n + kTb - 1) / kTb, own_max = (nb + kTvCtas - 1) / kTvCtas;
    uint64_t *bar = reinterpret_cast<uint64_t *>(raw + ((sizeof(TrsvShared) + 15) & ~size_t(15)));  // [2][nb]
    double *y = reinterpret_cast<double *>(bar + 2 * nb);                                           // [nb][32]
    double *rhs = y + (size_t)nb * kTb;                                                             // [own_max][32]
    int *perm = reinterpret_cast<int *>(y);                                                         // [n], before y
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int c = blockIdx.x % kTvCtas;
    B += blockIdx.x / kTvCtas;
    for (int e = t; e < 2 * nb; e += kTvThreads) {
        mbar_init(&bar[e], 1);
    }
    if (t == 0) S.err = 0;
    for (int r = t; r < n; r += kTvThreads) perm[r] = r;
    __syncthreads();
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int e = t; e < 2 * nb; e += kTvThreads) expect_tx(&bar[e], kTb * 8);
    // the row order: each warp works out the net effect of 64 interchanges on the at most 128 rows they
    // touch (traced backwards, a lane per slot), then the blocks are applied in order
    for (int k0 = 0; k0 < n; k0 += kTvWarps * kSwapBlock) {
        const int q0 = k0 + warp * kSwapBlock, cnt = min(kSwapBlock, n - q0);
        if (cnt > 0) {
            int *piv = S.piv[warp];
            for (int q = lane; q < kSwapBlock; q += 32) piv[q] = q < cnt ? ipiv[q0 + q] : -1;
            __syncwarp();
            int d[4], r[4];
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const int q = (s & 1) * 32 + lane;
                d[s] = q >= cnt ? -1 : s < 2 ? q0 + q : piv[q] >= q0 + cnt ? piv[q] : -1;
            }
#pragma unroll
            for (int s = 2; s < 4; s++) {
                const int q = (s & 1) * 32 + lane;
                for (int p = 0; p < cnt; p++)
                    if (p < q && piv[p] == d[s]) d[s] = -1;
            }
#pragma unroll
            for (int s = 0; s < 4; s++) r[s] = d[s];
            for (int p = cnt - 1; p >= 0; p--) {
                const int a = q0 + p, b = piv[p];
#pragma unroll
                for (int s = 0; s < 4; s++) r[s] = r[s] == a ? b : r[s] == b ? a : r[s];
            }
#pragma unroll
            for (int s = 0; s < 4; s++) S.dst[warp][s * 32 + lane] = d[s], S.src[warp][s * 32 + lane] = r[s];
        }
        __syncthreads();
        for (int w = 0; w < kTvWarps && k0 + w * kSwapBlock < n; w++) {
            int v = 0, d = -1;
            if (t < 2 * kSwapBlock) {
                d = S.dst[w][t];
                if (d >= 0) v = perm[S.src[w][t]];
            }
            __syncthreads();
            if (d >= 0) perm[d] = v;
            __syncthreads();
        }
    }
    for (int e = t; e < own_max * kTb; e += kTvThreads) {
        const int b = (e / kTb) * kTvCtas + c, r = b * kTb + e % kTb;
        rhs[e] = b < nb && r < n ? B[(int64_t)perm[r] * ldb] : 0.0;
    }
    cluster_sync();  // every CTA's mbarriers are armed, its permutation read, and all of b

    for (int pass = 0; pass < 2; pass++) {
        const bool up = pass == 1;
        uint64_t *pb = bar + pass * nb;
        // owned blocks in the order of the pass; p: position of a block in that order
        const int last = nb - 1;
        for (int k = 0; k < own_max; k++) {
            const int own = up ? own_max - 1 - k : k, b = own * kTvCtas + c;
            if (b >= nb) continue;
            const int np = up ? last - b : b;  // blocks before this one
            auto block = [&](int p) { return up ? last - p : p; };
            const int row = b * kTb + lane;
            const double *A = LU + (int64_t)min(row, n - 1) * ld;
            for (int e = t; e < kTb * kTb; e += kTvThreads) {  // the diagonal block, the identity beyond row n
                const int i = e / kTb, q = e % kTb, gr = b * kTb + i, gc = b * kTb + q;
                S.T[i][q] = gr < n && gc < n ? LU[(int64_t)gr * ld + gc] : (i == q ? 1.0 : 0.0);
            }
            // all blocks but the previous one: eight warps, four columns each, four blocks' loads in flight
            double acc = 0.0;
            const int cw = warp * 4;
            for (int p0 = 0; p0 + 1 < np; p0 += 4) {
                double m[4][4];
#pragma unroll
                for (int s = 0; s < 4; s++) {
                    const int p = min(p0 + s, np - 1), j = block(p);
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int col = j * kTb + cw + q;
                        m[s][q] = col < n ? A[col] : 0.0;
                    }
                }
#pragma unroll
                for (int s = 0; s < 4; s++)
                    if (p0 + s + 1 < np) {
                        const int j = block(p0 + s);
                        cluster_wait(&pb[j], 0, &S.err, kWaitLimitNs);
#pragma unroll
                        for (int q = 0; q < 4; q++) acc = fma(m[s][q], y[j * kTb + cw + q], acc);
                    }
            }
            S.ps[warp][lane] = acc;
            // the previous block's slice: four warps, eight columns each
            double ml[8];
            const int jl = np > 0 ? block(np - 1) : 0;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int col = jl * kTb + warp * 8 + q;
                ml[q] = np > 0 && warp < 4 && col < n ? A[col] : 0.0;
            }
            __syncthreads();
            double v = 0.0, tr[kTb], rd = 1.0;
            bool divide = false;
            if (warp == 0) {
                v = up ? y[b * kTb + lane] : rhs[own * kTb + lane];
#pragma unroll
                for (int w = 0; w < kTvWarps; w++) v -= S.ps[w][lane];
#pragma unroll
                for (int q = 0; q < kTb; q++) tr[q] = S.T[lane][q];
                if (up) {  // T x = T D^-1 (D x): the columns scaled ahead take the multiplication off the chain
                    const int ex = (__double2hiint(S.T[lane][lane]) >> 20) & 0x7ff;
                    bool bad = ex < 64 || ex > 1982;
                    rd = __drcp_rn(S.T[lane][lane]);
#pragma unroll
                    for (int q = 0; q < kTb; q++) {
                        const double t0 = tr[q];
                        tr[q] *= __shfl_sync(0xffffffffu, rd, q);
                        const int hi = __double2hiint(tr[q]), e = (hi >> 20) & 0x7ff;
                        bad = bad || (q > lane && (e == 0x7ff || (e == 0 && t0 != 0.0)));
                    }
                    // a reciprocal or a scaled entry outside the normal range loses accuracy, or is infinite: divide there
                    divide = __any_sync(0xffffffffu, bad);
                }
            }
            if (np > 0) {
                if (warp < 4) {
                    cluster_wait(&pb[jl], 0, &S.err, kWaitLimitNs);
                    double a = 0.0;
#pragma unroll
                    for (int q = 0; q < 8; q++) a = fma(ml[q], y[jl * kTb + warp * 8 + q], a);
                    S.pl[warp][lane] = a;
                }
                __syncthreads();
            }
            if (warp == 0) {
                if (row >= n) v = 0.0;
                else if (np > 0) v -= (S.pl[0][lane] + S.pl[1][lane]) + (S.pl[2][lane] + S.pl[3][lane]);
                if (!up) {
#pragma unroll
                    for (int q = 0; q < kTb - 1; q++) {
                        const double yq = __shfl_sync(0xffffffffu, v, q);
                        const double w = fma(-tr[q], yq, v);
                        v = lane > q ? w : v;
                    }
                } else {
                    if (divide) {
                        for (int q = kTb - 1; q >= 0; q--) {
                            const double x = v / S.T[lane][lane];
                            const double xq = __shfl_sync(0xffffffffu, x, q);
                            const double w = fma(-S.T[lane][q], xq, v);
                            v = lane == q ? x : lane < q ? w : v;
                        }
                    } else {
#pragma unroll
                        for (int q = kTb - 1; q > 0; q--) {
                            const double vq = __shfl_sync(0xffffffffu, v, q);
                            const double w = fma(-tr[q], vq, v);
                            v = lane < q ? w : v;
                        }
                        v *= rd;
                    }
                }
                S.out[lane] = *(volatile int *)&S.err ? __longlong_as_double(0x7ff8000000000000ll) : v;
            }
            __syncthreads();
            const double o = S.out[lane];
#pragma unroll
            for (int d = 0; d < kTvCtas / kTvWarps; d++)
                send(&y[b * kTb + lane], &pb[b], warp + d * kTvWarps, o);
            if (up && warp == 0 && row < n) B[(int64_t)row * ldb] = o;
        }
        // Every value sent to this CTA has arrived before any CTA goes on: nothing orders two st.async to one
        // address, so a forward value still under way could land on the backward one that replaces it
        // (a CTA waits for a block by itself only where it needs the block), and a CTA that has
        // ended must not be a store's target.
        for (int e = t; e < nb; e += kTvThreads) cluster_wait(&pb[e], 0, &S.err, kWaitLimitNs);
        __syncthreads();
        cluster_sync();
    }
    // a wait that ran out: the results behind it are NaN
    if (t == 0 && S.err && err) atomicExch(err, 1);
}

static size_t trsv_smem(int64_t n) {
    const size_t nb = (size_t)ceil_div(n, kTb), own = (size_t)ceil_div(nb, kTvCtas);
    return ((sizeof(TrsvShared) + 15) & ~size_t(15)) + 16 * nb + 8 * kTb * (nb + own);
}
bool trsv_fits(int64_t n) { return trsv_smem(n) <= 232448; }

int trsv_cluster(int64_t n, int64_t nrhs, const double *LU, int64_t ld, const int32_t *ipiv, double *B, int64_t ldb,
                 int *err, cudaStream_t st) {
    FLG_ONCE_PER_DEVICE(
        FLG_CUDA(cudaFuncSetAttribute(trsv_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        FLG_CUDA(cudaFuncSetAttribute(trsv_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448)));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(kTvCtas * nrhs));
    cfg.blockDim = dim3(kTvThreads);
    cfg.dynamicSmemBytes = trsv_smem(n);
    cfg.stream = st;
    cudaLaunchAttribute at[1] = {};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kTvCtas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    FLG_CUDA(cudaLaunchKernelEx(&cfg, trsv_cluster_kernel, LU, ld, ipiv, B, ldb, (int)n, err));
    count_launch();
    return FLG_OK;
}

}  // namespace flg
