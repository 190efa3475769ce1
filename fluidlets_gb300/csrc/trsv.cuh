// trsv.cuh -- interface of the one-launch triangular solves (trsv.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace flg {

bool trsv_fits(int64_t n);  // the solution and the mbarriers fit the shared memory of a CTA
int trsv_cluster(int64_t n, int64_t nrhs, const double *LU, int64_t ld, const int32_t *ipiv, double *B, int64_t ldb,
                 int *err, cudaStream_t st);

}  // namespace flg
