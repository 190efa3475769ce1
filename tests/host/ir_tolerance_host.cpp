// The refinement's step rule compiled for the host, for tests/test_ir_tolerance.py.
#include "../../fluidlets_gb300/csrc/ir_tolerance.cuh"

extern "C" double ir_inner(double tol, double rn) { return flg::ir_inner_tolerance(tol, rn); }
extern "C" int ir_done(double tol, double rn, int beyond) { return flg::ir_done(tol, rn, beyond != 0); }
