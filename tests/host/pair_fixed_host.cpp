// The fixed-point pair functions compiled for the host, for tests/test_pair_fixed.py.
#include "../../fluidlets_gb300/csrc/pair_fixed.cuh"

using namespace flg;

// coefficients a, b1, b2, c, z of the wall block from (0, 0, h) with blob width e to (x, y, t), times t h
extern "C" void wall_block(double x, double y, double t, double h, double e, double *out) {
    const double rq = fma(y, y, fma(x, x, e * e)), dm = t - h, dp = t + h;
    const FxWallBlock w = fx_wall_block(dm, dp, fma(dm, dm, rq), fma(dp, dp, rq), e, fx_const(t), fx_const(h));
    out[0] = w.a, out[1] = w.b1, out[2] = w.b2, out[3] = w.c, out[4] = w.z;
}
// coefficients of G = A I + B d d^T; kind 0: Stokeslet, 1: Brinkman with alpha
extern "C" void radial_block(int kind, double x, double y, double z, double e, double alpha, double *out) {
    const double Q = fma(z, z, fma(y, y, fma(x, x, e * e)));
    const FxDir g = fx_dir(Q, e);
    fx_radial_block(g, kind == 0 ? fx_stokeslet(g) : fx_brinkman(g, fx_alpha(alpha)), fx_const(1.0), out, out + 1);
}
