// ir_tolerance.cuh -- how far the steps of the dense refinement go (krylov.cu, ir_graph.cu).
#pragma once
#include <math.h>

#if defined(__CUDACC__)
#define FLG_IR_HD __host__ __device__
#else
#define FLG_IR_HD
#endif

namespace flg {

// Inner (preconditioned) tolerance of a step at residual norm rn, aimed at tol.  At 1e-4 many
// inner solves ended just below it after one iteration, and a third FP64 residual was needed (wall, 8,192
// blobs, tf32: 3 steps, 45.4 ms); at 1e-6 two steps reach 1e-12 (42.1 ms).  A step gains eight digits at most (its
// operator is the FP32 copy of the matrix); one that needs no more than that aims at a fiftieth of tol, as far as
// those eight digits go.
FLG_IR_HD inline double ir_inner_tolerance(double tol, double rn) {
    const double need = tol / rn;
    if (need >= 1.0) return 1e-4;  // (a step beyond the tolerance, see below)
    if (!(need >= 1e-8)) return 1e-6;
    return fmin(1e-6, fmax(0.02 * need, 2e-8));
}

// Whether the refinement is done at residual norm rn.  The error of the solution is the residual times the condition
// number, and two steps end anywhere below tol where ones of 1e-4 had overshot it (swimmer of 1,470 unknowns: residual
// 2.5e-13, forces exact to 5e-11 instead of 9e-14): above 3 % of tol one more step follows.  Largest errors over 60
// bodies and 14 swimmers, steps of 1e-4: 1.0e-12, 5.1e-13; these with the limit at 5 % 3.6e-13, 2.3e-12, at 3 % 2.7e-13,
// 5.1e-13, at 2 % 2.0e-13, 5.1e-13.  Two steps leave spheres and walls at 1.1 to 2.6 % (the FP32 copy's rounding squared),
// so that at 2 % a third of them, at 1 % nearly all take a third step: 1,536 blobs 3.1 -> 3.7 ms.
FLG_IR_HD inline bool ir_done(double tol, double rn, bool beyond) { return rn <= tol && (beyond || rn <= 0.03 * tol); }

}  // namespace flg
