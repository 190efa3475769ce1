// panel.cuh -- interface of the cluster panel of the FP64 LU (panel.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace flg {

constexpr int kHalf = 32;        // panel width: half of a 64-column block
constexpr int kPanelCtas = 16;   // CTAs of the cluster
constexpr int64_t kClusterPanelRows = kPanelCtas * 32 * 16;  // 8,192 rows

struct ClusterPanelArgs {
    double *A;
    int64_t ld, n, k0;
    int kb;
    int32_t *ipiv;
    int *info;      // 1 + first zero or non-finite pivot
    int *err;       // raised by a timed-out wait
    int cc0, cc1;   // companion columns that receive the interchanges ...
    int trsm;       // ... and U12 = L11^-1 A12
    int rpc;        // rows per CTA (set by cluster_panel)
};

int cluster_panel(const ClusterPanelArgs &a, cudaEvent_t started, cudaStream_t st);
int half_update(double *A, int64_t ld, int64_t r0, int64_t n, int64_t k0, int nc, cudaStream_t st);

}  // namespace flg
