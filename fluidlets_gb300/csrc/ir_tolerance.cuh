// ir_tolerance.cuh -- how far the steps of the dense refinement go (krylov.cu, ir_graph.cu).
#pragma once
#include <math.h>

#if defined(__CUDACC__)
#define FLG_IR_HD __host__ __device__
#else
#define FLG_IR_HD
#endif

namespace flg {

// A step's inner (preconditioned) tolerance, and the residual norm at which it stops after k columns: a hundredth of
// it after the first column, which often ends just below it, so that a third step, with its FP64 residual, would be
// needed for digits that a second column gives (wall, 8,192 blobs, tf32: 45.4 ms, 42.1 with two).  1e-6
// throughout takes more columns than it is worth where each gains less (swimmer of 1,206 unknowns: 12 columns in two
// steps, 2.32 ms and a residual of 7e-13; this way 8 in three, 1.75 ms and 4e-15).
constexpr double kIrInner = 1e-4;
FLG_IR_HD inline double ir_inner_limit(double ptol, int k) { return k <= 1 ? 1e-2 * ptol : ptol; }

// Whether the refinement is done at residual norm rn.  The error of the solution is the residual times the condition
// number, and the steps end anywhere below tol: above 5 % of it one more follows.  Largest errors over 60 bodies and 14
// swimmers: 3.6e-13, 5.5e-13 (without the step 3.6e-13, 2.8e-12; by steps of 1e-4 throughout 1.0e-12, 5.1e-13).
// Two steps leave spheres and walls at 1.1 to 2.9 % (the FP32 copy's rounding squared), and they need no third.
FLG_IR_HD inline bool ir_done(double tol, double rn, bool beyond) { return rn <= tol && (beyond || rn <= 0.05 * tol); }

}  // namespace flg
