// The refinement's step rules compiled for the host, for tests/test_ir_tolerance.py.
#include "../../fluidlets_gb300/csrc/ir_tolerance.cuh"

extern "C" double ir_limit(double beta, int k) { return flg::ir_inner_limit(flg::kIrInner * beta, k); }
extern "C" int ir_done(double tol, double rn, int beyond) { return flg::ir_done(tol, rn, beyond != 0); }
