// pair_fixed.cuh -- the FP64 pair kernels' coefficients in 60-bit fixed point (fixed.cuh).
//
// The same formulas as pair_math.cuh's, the coefficients written in bounded quantities.  With Q = |d|^2 + e^2 =
// q 2^(2E), y = q^-1/2, s = Q^-1/2 = y 2^-E and w = e s:
//   Stokeslet     8 pi u = A f + B (f.d) d,  A = s (1 + w^2), B = s^3
//   Brinkmanlet   4 pi u = A f + B (f.d) d,  A = s (f1 + w^2 f2), B = s^3 f2         below z = 1/2 (series), and
//                        A = s^3 / alpha^2 (F1 + w^2 F2), B = s^5 / alpha^2 F2, F = z^2 f, above:
//     F1 = E (1 + z + z^2) - 1, F2 = 3 - E (3 + 3 z + z^2), E = e^-z from 2^-n 2^(-i/64) e^-x with a table
//     (P. T. P. Tang, "Table-driven implementation of the exponential function in IEEE
//     floating-point arithmetic", ACM TOMS 15, 1989)
//   wall          8 pi u_j = 2 t h sF s^2 [c f_j + d_j sF^2 (Z3 (f.d) + 3 rho^3 (D - dp f_z))]      (j = x, y)
//                 8 pi u_z = 2 t h sF s^2 [z f_z + D sF^2 (Z3 dm + 3 rho^3 dp)]
//     with rho = s / sF <= 1 (s of the image), D = d_x f_x + d_y f_y, dm = t - h, dp = t + h,
//     Z1 = 2 / (1 + rho), Z3 = Z1 (1 + rho + rho^2) = 2 + ... , c = Z1 + w^2 Z3 - rho + 3 w^2 rho^3,
//     z = Z1 + w^2 Z3 - rho - 3 w^2 rho^3 + Z3 n^2 - 3 rho nI^2, n = dm sF, nI = dp s
//   (the bracket is the image form of pair_math.cuh divided by sF^3 rho^2, which keeps its
//   precision where the wall is far: rho -> 0).
// A coefficient is a double of 2^-54 relative accuracy or better (of its terms, where they cancel).  Displacements,
// Q, and the products with displacement and strength stay in FP64, so that every component of a
// velocity keeps the precision of an FP64 sum of its own terms: a component may be small beside the
// others, as may the displacement along it, and fixed point against a common exponent would round
// it to 2^-58 of the largest.  (The Stokeslet's sums are integers with an exponent for each component.)
// Pairs outside the ranges (Q not a normal number far from the limits, targets and sources on
// opposite sides of the wall) go to the FP64 functions, pair by pair.
#pragma once
#include "fixed.cuh"

namespace flg {

// exponents of Q that the fixed-point path takes: every exponent sum stays far inside the range, and so do the
// coefficients (s^3 of a radial kernel's sum, with one height s^4 of the wall's)
constexpr int kQExpMax = 1000, kQExpRadial = 640, kQExpWall = 360;
FLG_HD bool q_in_range(double Q, int limit = kQExpMax) {
    const int ex = (int)(dbits(Q) >> 52);  // (a sign bit makes it too large)
    return ex >= 1023 - limit && ex <= 1023 + limit;
}

// what the pair kernels give: u = (A f + B (f.n) n) 2^x of a radial kernel, n = d / sqrt(Q)
struct FxRadial {
    q60 A, B;  // A in [-1.8, 1.8], B in [0, 1.6]
    int x;
};
struct FxDir {  // the root and w^2
    q60 w2;
    QRsqrt r;
};
FLG_HD FxDir fx_dir(double Q, double e) {
    FxDir g;
    g.r = q_rsqrt(Q);
    const Qf w = qf(qmul(qf(q_mag(e, g.r.e)), qf(g.r.y)));
    g.w2 = qmul(w, w);
    return g;
}

FLG_HD FxRadial fx_stokeslet(const FxDir &g) {
    // (1 + w^2) / 2 and 1 / 2 of the root
    FxRadial r;
    r.A = qmul(qf((kQ1 + g.w2) >> 1), qf(g.r.y));
    r.B = g.r.y >> 1;
    r.x = 1 - (g.r.e - 1023);
    return r;
}

// alpha = am 2^ae with am in [1/2, 1); 1 / alpha^2 = ia 2^iae with ia in [1/2, 1)
struct FxAlpha {
    q60 am, ia;
    int ae, iae;
};
inline FxAlpha fx_alpha(double alpha) {
    FxAlpha a;
    if (alpha == 0.0) return {0, 0, -(1 << 20), 0};  // the series at z = 0
    int e;
    const double m = std::frexp(alpha < 1.7e308 ? alpha : 1.7e308, &e);  // (an infinite alpha: u = 0)
    a.am = (q60)std::ldexp(m, 60);
    a.ae = e;
    const long double i = 1.0L / ((long double)m * m);  // in (1, 4]
    int ie;
    const long double im = std::frexp(i, &ie);
    a.ia = (q60)std::ldexp(im, 60);
    a.iae = ie - 2 * e;
    return a;
}

// 2^(-i / 64)
#define FLG_EXP_TABLE \
    0x1000000000000000ll, 0x0fd3e0c0cf486c17ll, 0x0fa83b2db722a034ll, 0x0f7d0df730ad13bcll, \
    0x0f5257d152486cc3ll, 0x0f281773c59ffb14ll, 0x0efe4b99bdcdaf5dll, 0x0ed4f301ed9942b8ll, \
    0x0eac0c6e7dd24393ll, 0x0e8396a503c4bdc7ll, 0x0e5b906e77c8348bll, 0x0e33f8972be8a5a5ll, \
    0x0e0ccdeec2a94e11ll, 0x0de60f4825e0e912ll, 0x0dbfbb797daf2375ll, 0x0d99d15c278afd7bll, \
    0x0d744fccad69d6afll, 0x0d4f35aabcfedfa2ll, 0x0d2a81d91f12ae46ll, 0x0d06333daef2b259ll, \
    0x0ce248c151f8480ell, 0x0cbec14fef2727c6ll, 0x0c9b9bd866e2f27all, 0x0c78d74c8abb9b16ll, \
    0x0c5672a115506daell, 0x0c346ccda2497640ll, 0x0c12c4cca6670945ll, 0x0bf1799b67a73108ll, \
    0x0bd08a39f580c36cll, 0x0baff5ab2133e460ll, 0x0b8fbaf4762fb9efll, 0x0b6fd91e328d1779ll, \
    0x0b504f333f9de648ll, 0x0b311c412a911249ll, 0x0b123f581d2ac259ll, 0x0af3b78ad690a437ll, \
    0x0ad583eea42a14acll, 0x0ab7a39b5a93ed33ll, 0x0a9a15ab4ea7c0f0ll, 0x0a7cd93b4e965357ll, \
    0x0a5fed6a9b15138fll, 0x0a43515ae09e680all, 0x0a27043030c49682ll, 0x0a0b0510fb9714fcll, \
    0x09ef5326091a111bll, 0x09d3ed9a72cffb75ll, 0x09b8d39b9d54e554ll, 0x099e0459320b7fa6ll, \
    0x09837f0518db8a97ll, 0x096942d3720185a0ll, 0x094f4efa8fef7096ll, 0x0935a2b2f13e6e93ll, \
    0x091c3d373ab11c33ll, 0x09031dc431466b1ell, 0x08ea4398b45cd53cll, 0x08d1adf5b7e5ba9ell, \
    0x08b95c1e3ea8bd6ell, 0x08a14d575496efdall, 0x088980e8092da852ll, 0x0871f61969e8d101ll, \
    0x085aac367cc487b1ll, 0x0843a28c3acde404ll, 0x082cd8698ac2ba1dll, 0x08164d1f3bc03077ll
// series coefficients of f1 and f2 (pair_math.cuh), 16 terms: the next is below 2^-60 at z = 1/2
#define FLG_BR_Q1 \
    576460752303423488ll, -768614336404564651ll, 432345564227567616ll, -153722867280912930ll, \
    40031996687737742ll, -8235153604334621ll, 1401119884070821ll, -203337126032954ll, \
    25734855013546ll, -2888311449332ll, 291238071141ll, -26661336455ll, \
    2235002907ll, -172804959ll, 12398315ll, -829796ll
#define FLG_BR_Q2 \
    576460752303423488ll, 0ll, -144115188075855872ll, 76861433640456465ll, \
    -24019198012642645ll, 5490102402889748ll, -1000799917193444ll, 152502844524715ll, \
    -20015998343869ll, 2310649159465ll, -238285694570ll, 22217780379ll, \
    -1891156306ll, 148118536ll, -10745206ll, 726071ll
#if defined(__CUDACC__)
static __constant__ q60 c_q_br1[16] = {FLG_BR_Q1};
static __constant__ q60 c_q_br2[16] = {FLG_BR_Q2};
static __device__ const q60 c_q_exp[64] = {FLG_EXP_TABLE};
#endif
static const q60 h_q_br1[16] = {FLG_BR_Q1};
static const q60 h_q_br2[16] = {FLG_BR_Q2};
static const q60 h_q_exp[64] = {FLG_EXP_TABLE};
FLG_HD q60 q_br1(int i) {
#if defined(__CUDA_ARCH__)
    return c_q_br1[i];
#else
    return h_q_br1[i];
#endif
}
FLG_HD q60 q_br2(int i) {
#if defined(__CUDA_ARCH__)
    return c_q_br2[i];
#else
    return h_q_br2[i];
#endif
}
FLG_HD q60 q_exp_table(int i) {
#if defined(__CUDA_ARCH__)
    return c_q_exp[i];
#else
    return h_q_exp[i];
#endif
}

// a b for b in Q36 below 2^30 (a factor below 1/64)
FLG_HD q60 qmul36(q60 a, int b) {
    const Qf f = qf(a);
    return (((q60)f.h * b) >> 6) + (((q60)f.l * b) >> 36);
}
// 2^-(v 2^kz) = m 2^-n, m in (1/2, 1], for v in [0, 1.45), 0 <= kz <= 7
FLG_HD q60 q_exp2neg(q60 v, int kz, int *n) {
    const q60 frac = (q60)((uint64_t)v << kz) & (kQ1 - 1);
    *n = (int)(v >> (60 - kz));
    const int i = (int)(frac >> 54);
    const q60 x = qmul(qf((frac << 6) & (kQ1 - 1)), qf(799144290325165979ll >> 6));  // remainder ln(2) / 64
    const int xs = (int)(x >> 24);
    const q60 v4 = (kQ1 / 24) - qmul36((kQ1 / 120) - qmul36((kQ1 / 720) - qmul36(kQ1 / 5040, xs), xs), xs);
    const Qf xf = qf(x);
    const q60 u = (kQ1 / 2) - qmul(xf, qf((kQ1 / 6) - qmul(xf, qf(v4))));
    const q60 p = kQ1 - x + qmul(qf(qmul(xf, xf)), qf(u));
    return qmul(qf(q_exp_table(i)), qf(p));
}
// e^-z for z = zm 2^kz with zm in [1/2, 1): zm log2(e) is in (0.7, 1.45)
FLG_HD q60 q_expneg(q60 zm, int kz, int *n) { return q_exp2neg(qmul(qf(zm), qf(1663314137230540311ll)), kz, n); }

// bits that |x| < 2 can move up so that the larger ones of or-ed x are in [1/2, 1); q_abs1 is |x| or |x| - 1
FLG_HD uint64_t q_abs1(q60 x) { return (uint64_t)(x ^ (x >> 63)); }
FLG_HD int q_room(uint64_t m) {
#if defined(__CUDA_ARCH__)
    const int lz = __clz((int)(m >> 32));
#else
    const int lz = (m >> 32) ? __builtin_clz((unsigned)(m >> 32)) : 32;
#endif
    return lz > 4 ? lz - 4 : 0;
}
FLG_HD q60 q_shift(q60 x, int s) {  // x 2^-s
    return s >= 0 ? x >> (s < 63 ? s : 63) : x << -s;
}

// |alpha| sqrt(Q) = m 2^k, m in [1/2, 1)
struct FxZ {
    q60 m;
    int k;
};
FLG_HD FxZ fx_z(const FxDir &g, q60 am, int ae) {
    const q60 zm = qmul(qf(am), qf(qmul(qf(g.r.qh), qf(g.r.y))));  // in [1/4, 1)
    const int low = zm < kQ1 / 2;
    return {zm << low, ae + (g.r.e - 1023) + 1 - low};
}
FLG_HD FxRadial fx_series(const FxDir &g, const FxZ &zz, const FxAlpha &) {  // k < 0
    const Qf y = qf(g.r.y), z = qf(q_shift(zz.m, -zz.k));
    q60 f1 = q_br1(15), f2 = q_br2(15);
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int n = 14; n >= 0; n--) {
        f1 = qmul(qf(f1), z) + q_br1(n);
        f2 = qmul(qf(f2), z) + q_br2(n);
    }
    FxRadial r;
    r.A = qmul(qf(f1 + qmul(qf(f2), qf(g.w2))), y);
    r.B = qmul(qf(f2), y);
    r.x = 1023 - g.r.e;
    return r;
}
FLG_HD FxRadial fx_closed(const FxDir &g, const FxZ &zz, const FxAlpha &al) {  // k >= 0
    const Qf y = qf(g.r.y);
    const int E = g.r.e - 1023, kz = zz.k;
    const q60 zm = zz.m;
    FxRadial r;
    q60 F1 = -kQ1, F2h = kQ1 + kQ1 / 2;  // F1, F2 / 2 where E has vanished
    if (kz < 6 || (kz == 6 && zm < kQ1 / 64 * 52)) {
        int n;
        const Qf em = qf(q_expneg(zm, kz, &n));
        const q60 z2 = qmul(qf(zm), qf(zm)), z1 = zm >> kz, z0 = kQ1 >> (2 * kz);  // over 4^kz
        const int h1 = kz == 0, h2 = kz < 2 ? 2 - kz : 0;  // so that the polynomials stay below 2
        F1 += q_shift(qmul(em, qf((z2 + z1 + z0) >> h1)), n - 2 * kz - h1);
        F2h -= q_shift(qmul(em, qf((z2 + 3 * (z1 + z0)) >> h2)), n - 2 * kz - h2 + 1);
    }
    // (small factors are scaled up: F1 and F2 of z < 1, y^3 / alpha^2 below 1/4)
    q60 k = qmul(qf(qmul(qf(qmul(y, y)), y)), qf(al.ia));
    const int sk = k < kQ1 / 4 ? 2 : 0, sf = kz == 0 ? 2 : 0;
    const Qf kf = qf(k << sk), f2 = qf(F2h << sf);
    r.A = qmul(qf(((F1 << sf) >> 1) + qmul(f2, qf(g.w2))), kf);
    r.B = qmul(f2, kf);
    // A and B up to [1/2, 1): a sum keeps its terms to 2^-58 of the largest exponent it has met
    const int s = q_room(q_abs1(r.A) | q_abs1(r.B));
    r.A <<= s, r.B <<= s;
    r.x = 1 + al.iae - 3 * E - sk - sf - s;
    return r;
}
FLG_HD FxRadial fx_brinkman(const FxDir &g, const FxAlpha &al) {
    const FxZ z = fx_z(g, al.am, al.ae);
    return z.k < 0 ? fx_series(g, z, al) : fx_closed(g, z, al);
}

// A and B of u = A f + B (f.d) d
struct FxCoef {
    double A, B;
};
FLG_HD FxCoef fx_coef(const FxDir &g, const FxRadial &r) {
    const Qf y = qf(g.r.y);
    return {q_to_double(r.A, r.x), q_to_double(qmul(qf(r.B), qf(qmul(y, y))), r.x - 2 * (g.r.e - 1023))};
}

// ---- Stokeslet sums in integers ---------------------------------------------------------------------
// A Stokeslet pair has so few operations that the ten FP64 products with displacement and strength would be what
// bounds its sum, so they are integers too, every component with an exponent of its own: strengths,
// displacement, and the sums, so that a component's rounding stays 2^-56 of its own largest term.
struct FxNum {
    q60 m;  // [1/2, 1), with the sign; 0 for zero
    int e;  // x = m 2^e
};
constexpr int kFxTiny = -(1 << 20);  // exponent of a zero
FLG_HD FxNum fx_num(double x) {      // (denormals count as zero)
    const uint64_t u = dbits(x);
    const int ex = (int)(u >> 52) & 0x7ff;
    if (ex == 0) return {0, kFxTiny};
    return {q_sign((q60)((u & 0x000fffffffffffffull) << 7 | 0x0800000000000000ull), d_neg(x)), ex - 1022};
}
FLG_HD bool fx_num_ok(double x) { return (dexp(x) != 0 || x == 0.0) && dexp(x) != 0x7ff; }
// Sums of three components over up to 32 terms m 2^x, |m| < 1: 64-bit integers of 57 fractional bits relative
// to the component's largest exponent so far, which outlives the 32 terms
struct FxAcc {
    q60 a[3];
    int x[3];
    FLG_HD void init() {
        clear();
        x[0] = x[1] = x[2] = -(1 << 24);
    }
    FLG_HD void clear() { a[0] = a[1] = a[2] = 0; }
    FLG_HD void add(int c, q60 m, int xt) {
        if (xt > x[c]) {  // makes room (rare once the first few terms have passed)
            const int s = xt - x[c] < 63 ? xt - x[c] : 63;
            a[c] >>= s;
            x[c] = xt;
        }
        const int s = x[c] - xt + 3 < 63 ? x[c] - xt + 3 : 63;
        a[c] += ((m >> (s - 1)) + 1) >> 1;
    }
    FLG_HD double value(int c) const { return q_to_double(a[c], x[c] + 3); }
};
// adds one pair's velocities of NF strengths f[3 NF] into acc[NF]
template <int NF>
FLG_HD void fx_add_stokeslet(double d0, double d1, double d2, double Q, double e, const FxNum *f, FxAcc *acc) {
    const FxDir g = fx_dir(Q, e);
    const int E = g.r.e - 1023;
    const Qf y = qf(g.r.y), A = qf(qmul(qf((kQ1 + g.w2) >> 1), y));  // (1 + w^2) s / 2
    const q60 y3 = qmul(qf(qmul(y, y)), y);
    const int n3 = q_room((uint64_t)y3);  // s^3 with its leading bit at 2^59
    const Qf B = qf(y3 << n3);
    const FxNum d[3] = {fx_num(d0), fx_num(d1), fx_num(d2)};
    const Qf D[3] = {qf(d[0].m), qf(d[1].m), qf(d[2].m)};
    for (int c = 0; c < NF; c++) {
        const FxNum *F = f + 3 * c;
        Qf Fm[3];
        q60 p[3];
        int xp[3];
        for (int k = 0; k < 3; k++) {
            Fm[k] = qf(F[k].m);
            p[k] = qmul(Fm[k], D[k]);
            xp[k] = F[k].e + d[k].e;
        }
        int xt = xp[0] > xp[1] ? xp[0] : xp[1];
        xt = (xt > xp[2] ? xt : xp[2]) + 2;  // f.d / 4 below 3/4
        q60 t = 0;
        for (int k = 0; k < 3; k++) t += p[k] >> (xt - xp[k] < 63 ? xt - xp[k] : 63);
        const Qf b = qf(qmul(qf(t), B));
        const int xb = xt - 3 * E - n3;
        for (int k = 0; k < 3; k++) {
            acc[c].add(k, qmul(A, Fm[k]), 1 - E + F[k].e);
            acc[c].add(k, qmul(b, D[k]), xb + d[k].e);
        }
    }
}

// ---- complex alpha --------------------------------------------------------------------------------
// The same functions of the complex z = |alpha| sqrt(Q) u, u = alpha / |alpha| (Re u >= 1/2, so that
// e^-z has vanished beside one from |z| = 128 on).  Imaginary parts carry an exponent of their own,
// xi, so that they keep their precision where z is small.
struct FxAlphaC {
    q60 am;        // |alpha| = am 2^ae, am in [1/2, 1)
    int ae, iae;   // 1 / alpha^2 = i 2^iae, |i| in [1/2, 1)
    q60 ur, ui;    // u
    q60 u2r, u2i;  // u^2
    q60 ir, ii;
    q60 cx, cy;    // Re(u) log2(e), Im(u) 2 / pi
};
// which alpha the fixed-point path takes: a finite one that decays, with an imaginary part that an
// absolute error of 2^-59 |alpha| still leaves its FP64 precision
inline bool fx_alpha_c_ok(double re, double im) {
    return std::fabs(re) < 1e150 && std::fabs(im) < 1e150 && re > 1e-150 && std::fabs(im) <= 1.7 * re &&
           std::fabs(im) >= re / 4;
}
inline FxAlphaC fx_alpha_c(double re, double im) {
    FxAlphaC a;
    const long double r = re, i = im, m2 = r * r + i * i, m = sqrtl(m2), ur = r / m, ui = i / m;
    auto q = [](long double x) { return (q60)llroundl(ldexpl(x, 60)); };
    int e;
    a.am = q(frexpl(m, &e));
    if (a.am >= kQ1) a.am = kQ1 - 1;
    a.ae = e;
    a.ur = q(ur), a.ui = q(ui);
    const long double u2r = ur * ur - ui * ui, u2i = 2 * ur * ui;
    a.u2r = q(u2r), a.u2i = q(u2i);
    const long double im2 = frexpl(1.0L / m2, &e);
    a.iae = e;
    a.ir = q(u2r * im2), a.ii = q(-u2i * im2);
    a.cx = q(ur * 1.442695040888963407359924681001892137L);
    a.cy = q(ui * 0.636619772367581343075535053490057448L);
    return a;
}

// cos and sin of 2 pi i / 64
struct alignas(16) QTrig {
    q60 c, s;
};
#define FLG_TRIG_TABLE \
    {1152921504606846976ll, 0ll}, {1147369872436662991ll, 113006068906017470ll}, \
    {1130768441178740757ll, 224923827593068887ll}, {1103277091691359535ll, 334675446864527722ll}, \
    {1065160580698383124ll, 441203958630471860ll}, {1016785991037278313ll, 543483435088187080ll}, \
    {958619196450722178ll, 640528868967736374ll}, {891220374967787610ll, 731405659690429196ll}, \
    {815238614083298888ll, 815238614083298888ll}, {731405659690429196ll, 891220374967787610ll}, \
    {640528868967736374ll, 958619196450722178ll}, {543483435088187080ll, 1016785991037278313ll}, \
    {441203958630471860ll, 1065160580698383124ll}, {334675446864527722ll, 1103277091691359535ll}, \
    {224923827593068887ll, 1130768441178740757ll}, {113006068906017470ll, 1147369872436662991ll}, \
    {0ll, 1152921504606846976ll}, {-113006068906017470ll, 1147369872436662991ll}, \
    {-224923827593068887ll, 1130768441178740757ll}, {-334675446864527722ll, 1103277091691359535ll}, \
    {-441203958630471860ll, 1065160580698383124ll}, {-543483435088187080ll, 1016785991037278313ll}, \
    {-640528868967736374ll, 958619196450722178ll}, {-731405659690429196ll, 891220374967787610ll}, \
    {-815238614083298888ll, 815238614083298888ll}, {-891220374967787610ll, 731405659690429196ll}, \
    {-958619196450722178ll, 640528868967736374ll}, {-1016785991037278313ll, 543483435088187080ll}, \
    {-1065160580698383124ll, 441203958630471860ll}, {-1103277091691359535ll, 334675446864527722ll}, \
    {-1130768441178740757ll, 224923827593068887ll}, {-1147369872436662991ll, 113006068906017470ll}, \
    {-1152921504606846976ll, 0ll}, {-1147369872436662991ll, -113006068906017470ll}, \
    {-1130768441178740757ll, -224923827593068887ll}, {-1103277091691359535ll, -334675446864527722ll}, \
    {-1065160580698383124ll, -441203958630471860ll}, {-1016785991037278313ll, -543483435088187080ll}, \
    {-958619196450722178ll, -640528868967736374ll}, {-891220374967787610ll, -731405659690429196ll}, \
    {-815238614083298888ll, -815238614083298888ll}, {-731405659690429196ll, -891220374967787610ll}, \
    {-640528868967736374ll, -958619196450722178ll}, {-543483435088187080ll, -1016785991037278313ll}, \
    {-441203958630471860ll, -1065160580698383124ll}, {-334675446864527722ll, -1103277091691359535ll}, \
    {-224923827593068887ll, -1130768441178740757ll}, {-113006068906017470ll, -1147369872436662991ll}, \
    {0ll, -1152921504606846976ll}, {113006068906017470ll, -1147369872436662991ll}, \
    {224923827593068887ll, -1130768441178740757ll}, {334675446864527722ll, -1103277091691359535ll}, \
    {441203958630471860ll, -1065160580698383124ll}, {543483435088187080ll, -1016785991037278313ll}, \
    {640528868967736374ll, -958619196450722178ll}, {731405659690429196ll, -891220374967787610ll}, \
    {815238614083298888ll, -815238614083298888ll}, {891220374967787610ll, -731405659690429196ll}, \
    {958619196450722178ll, -640528868967736374ll}, {1016785991037278313ll, -543483435088187080ll}, \
    {1065160580698383124ll, -441203958630471860ll}, {1103277091691359535ll, -334675446864527722ll}, \
    {1130768441178740757ll, -224923827593068887ll}, {1147369872436662991ll, -113006068906017470ll}
#if defined(__CUDACC__)
static __device__ const QTrig c_q_trig[64] = {FLG_TRIG_TABLE};
#endif
static const QTrig h_q_trig[64] = {FLG_TRIG_TABLE};
FLG_HD QTrig q_trig_table(int i) {
#if defined(__CUDA_ARCH__)
    const longlong2 v = *reinterpret_cast<const longlong2 *>(&c_q_trig[i]);
    return {v.x, v.y};
#else
    return h_q_trig[i];
#endif
}
// cos and sin of v quarter turns (v in Q60, any multiple of a whole turn may be missing): the
// nearest of 64 angles and Taylor polynomials of the rest, at most pi / 64
FLG_HD QTrig q_cos_sin(q60 v) {
    const q60 k = (q60)((uint64_t)v + (1ull << 55)) >> 56;  // sixteenths of a quarter turn
    const q60 rem = (q60)((uint64_t)v - ((uint64_t)k << 56));
    const Qf x = qf(qmul(qf(rem << 4), qf(113187804032455044ll)));
    const q60 x2 = qmul(x, x);
    const int s2 = (int)(x2 >> 24);
    const q60 s4 = (kQ1 / 120) - qmul36((kQ1 / 5040) - qmul36(kQ1 / 362880, s2), s2);
    const q60 c4 = (kQ1 / 24) - qmul36((kQ1 / 720) - qmul36(kQ1 / 40320, s2), s2);
    const Qf xf2 = qf(x2);
    // sin x = x - x^3 (1/6 - x^2 s4), cos x = 1 - x^2 (1/2 - x^2 c4)
    const q60 sn = qmul(x, qf(kQ1 - qmul(xf2, qf((kQ1 / 6) - qmul(xf2, qf(s4))))));
    const q60 cs1 = qmul(xf2, qf((kQ1 / 2) - qmul(xf2, qf(c4))));  // 1 - cos x
    const QTrig t = q_trig_table((int)k & 63);
    const Qf tc = qf(t.c), ts = qf(t.s), sf = qf(sn), cf = qf(cs1);
    return {t.c - qmul(tc, cf) - qmul(ts, sf), t.s - qmul(ts, cf) + qmul(tc, sf)};
}

// u = (A f + B (f.n) n) 2^x, A = (Ar + i Ai 2^xi), B alike; all below 1.5
struct FxRadialC {
    q60 Ar, Br, Ai, Bi;
    int x, xi;
};
FLG_HD FxRadialC fx_series(const FxDir &g, const FxZ &zz, const FxAlphaC &al) {
    const Qf y = qf(g.r.y), w2 = qf(g.w2), zf = qf(zz.m), ui = qf(al.ui);
    const q60 zm = zz.m;
    const int kz = zz.k;
    FxRadialC r;
    // a polynomial with real coefficients at a complex point: b_k = a_k + 2 Re(z) b_{k+1} - |z|^2 b_{k+2}
    const q60 zq = q_shift(zm, -kz), zr = qmul(qf(zq), qf(al.ur));
    const Qf p = qf(2 * zr), m = qf(qmul(qf(zq), qf(zq)));
    q60 b1 = q_br1(15), c1 = 0, b2 = q_br2(15), c2 = 0;
#if defined(__CUDA_ARCH__)
#pragma unroll 1  // unrolled, the pair outgrows the instruction cache: 4,099 x 2,500 1.81 ms, not 1.56
#endif
    for (int n = 14; n >= 1; n--) {
        const Qf h1 = qf(b1), h2 = qf(b2);
        const q60 t1 = q_br1(n) + qmul(h1, p) - qmul(qf(c1), m), t2 = q_br2(n) + qmul(h2, p) - qmul(qf(c2), m);
        c1 = b1, b1 = t1;
        c2 = b2, b2 = t2;
    }
    const Qf z0 = qf(zr), h1 = qf(b1), h2 = qf(b2);
    const q60 f1 = q_br1(0) + qmul(h1, z0) - qmul(qf(c1), m), f2 = q_br2(0) + qmul(h2, z0) - qmul(qf(c2), m);
    const Qf zi = qf(qmul(qf(qmul(zf, ui)), y));  // Im(z) y 2^-kz
    r.Ar = qmul(qf(f1 + qmul(qf(f2), w2)), y);
    r.Br = qmul(qf(f2), y);
    r.Ai = qmul(qf(b1 + qmul(h2, w2)), zi);
    r.Bi = qmul(h2, zi);
    r.x = 1023 - g.r.e;
    r.xi = kz;
    return r;
}
FLG_HD FxRadialC fx_closed(const FxDir &g, const FxZ &zz, const FxAlphaC &al) {
    const Qf y = qf(g.r.y), w2 = qf(g.w2), zf = qf(zz.m), ui = qf(al.ui);
    const int E = g.r.e - 1023, kz = zz.k;
    FxRadialC r;
    // F1 and F2 over 2^sc: below 1 at |z| < 1, up to 4 and 7 above
    const int sc = kz == 0 ? 0 : 3;
    q60 F1r = -(kQ1 >> sc), F1i = 0, F2r = 3 * (kQ1 >> sc), F2i = 0;
    if (kz < 8) {
        const q60 v = qmul(zf, qf(al.cx));  // Re(z) log2(e) 2^-kz
        int n;
        const Qf em = qf(q_exp2neg(v, kz, &n));
        const QTrig t = q_cos_sin((q60)((uint64_t)qmul(zf, qf(al.cy)) << kz));
        const Qf er = qf(qmul(em, qf(t.c))), ei = qf(-qmul(em, qf(t.s)));
        // 1 + z + z^2 and 3 + 3 z + z^2 over 4^kz 2^h
        const Qf zz = qf(qmul(zf, zf));
        const q60 z2r = qmul(zz, qf(al.u2r)), z2i = qmul(zz, qf(al.u2i));
        const q60 z1r = qmul(zf, qf(al.ur)) >> kz, z1i = qmul(zf, ui) >> kz, z0 = kQ1 >> (2 * kz);
        const int h1 = kz == 0, h2 = kz < 2 ? 2 - kz : 0;
        const Qf pr = qf((z2r + z1r + z0) >> h1), pi = qf((z2i + z1i) >> h1);
        const Qf qr = qf((z2r + 3 * (z1r + z0)) >> h2), qi = qf((z2i + 3 * z1i) >> h2);
        const int s1 = n - 2 * kz - h1 + sc, s2 = n - 2 * kz - h2 + sc;
        F1r += q_shift(qmul(er, pr) - qmul(ei, pi), s1);
        F1i += q_shift(qmul(er, pi) + qmul(ei, pr), s1);
        F2r -= q_shift(qmul(er, qr) - qmul(ei, qi), s2);
        F2i -= q_shift(qmul(er, qi) + qmul(ei, qr), s2);
    }
    const q60 y3 = qmul(qf(qmul(y, y)), y);
    const int s3 = y3 < kQ1 / 4 ? 2 : 0;
    const Qf y3f = qf(y3 << s3);
    const Qf kr = qf(qmul(y3f, qf(al.ir))), ki = qf(qmul(y3f, qf(al.ii))), f2r = qf(F2r), f2i = qf(F2i);
    const Qf ar = qf(F1r + qmul(f2r, w2)), ai = qf(F1i + qmul(f2i, w2));
    r.Ar = qmul(ar, kr) - qmul(ai, ki);
    r.Ai = qmul(ar, ki) + qmul(ai, kr);
    r.Br = qmul(f2r, kr) - qmul(f2i, ki);
    r.Bi = qmul(f2r, ki) + qmul(f2i, kr);
    const int s = q_room(q_abs1(r.Ar) | q_abs1(r.Ai) | q_abs1(r.Br) | q_abs1(r.Bi));  // as in fx_brinkman
    r.Ar <<= s, r.Ai <<= s, r.Br <<= s, r.Bi <<= s;
    r.x = sc + al.iae - 3 * E - s3 - s;
    r.xi = 0;
    return r;
}
FLG_HD FxRadialC fx_brinkman(const FxDir &g, const FxAlphaC &al) {
    const FxZ z = fx_z(g, al.am, al.ae);
    return z.k < 0 ? fx_series(g, z, al) : fx_closed(g, z, al);
}

struct FxCoefC {
    double Ar, Ai, Br, Bi;
};
FLG_HD FxCoefC fx_coef(const FxDir &g, const FxRadialC &r) {
    const Qf y = qf(g.r.y), y2 = qf(qmul(y, y));
    const int x = r.x - 2 * (g.r.e - 1023);
    return {q_to_double(r.Ar, r.x), q_to_double(r.Ai, r.x + r.xi), q_to_double(qmul(qf(r.Br), y2), x),
            q_to_double(qmul(qf(r.Bi), y2), x + r.xi)};
}

// a real factor c = m 2^x with |m| in [1/2, 1) (0 for c = 0)
struct FxConst {
    q60 m;
    int x;
};
FLG_HD FxConst fx_const(double c) {  // (not for denormals, infinities or NaN)
    if (c == 0.0) return {0, 0};
    const int e = dexp(c);
    return {q_of(c, e) >> 1, e - 1022};
}
FLG_HD bool fx_const_ok(double c) { return c == 0.0 || (dexp(c) > 64 && dexp(c) < 1982); }

// wall, times a factor k 2^kx (|k| in [1/4, 1) or 0): P = Z3, R = 3 rho^3 and their sum a (with the factor
// sF^2), c and z of the header.
// Where dm and dp are small beside the distance, P dm and R dp in FP64 keep their precision.  (As fixed-point n
// and nI, to 2^-60 of the distance, the xz entries were exact to 5e-13 at heights of 1e-6 of it.)
struct FxWall {
    double P, R, a, c, z;
};
FLG_HD FxWall fx_wall(double dm, double dp, double QF, double QI, double e, q60 k, int kx) {
    const FxDir f = fx_dir(QF, e);
    const QRsqrt i = q_rsqrt(QI);
    const Qf yI = qf(i.y), yF = qf(f.r.y), nm = qf(qmul(qf(q_mag(dm, f.r.e)), yF)), nI = qf(qmul(qf(q_mag(dp, i.e)), yI));
    // rho = (yI / yF) 2^(EF - EI), 1 / yF = q yF
    const q60 half = qmul(yI, qf(qmul(qf(f.r.qh), yF)));
    q60 r = q_shift(half << 1, i.e - f.r.e);
    if (r > kQ1) r = kQ1;
    // rho^3 with its relative precision where rho is small: r3 2^r3x, r3 in [1/8, 1)
    const int low = half < kQ1 / 2;  // (1/4 < half < 1)
    const Qf rho = qf(r), rm = qf(half << low);
    const q60 r3 = qmul(rm, qf(qmul(rm, rm)));
    const int r3x = 3 * (1 - low - (i.e - f.r.e));
    const q60 rho2 = qmul(rho, rho);
    const q60 Z1h = q_rcp1p(r);  // Z1 / 2
    const q60 Z3h = kQ1 + qmul(qf(rho2), qf(Z1h));  // Z3 / 2 = 1 + rho^2 / (1 + rho)
    const q60 rho3 = qmul(qf(rho2), rho), w2r3 = qmul(qf(f.w2), qf(rho3));
    const q60 base = Z1h + qmul(qf(f.w2), qf(Z3h)) - qhalf(r), i3 = w2r3 + qhalf(w2r3);
    const q60 c4 = qhalf(base + i3);  // c / 4
    const q60 rn2 = qmul(rho, qf(qmul(nI, nI)));
    const q60 z4 = qhalf(base - i3) + qhalf(qmul(nm, qf(qmul(qf(Z3h), nm))) - rn2 - qhalf(rn2));
    // the common factor k sF s^2, scaled up to [1/2, 1)
    q60 g = qmul(qf(qmul(yF, qf(qmul(yI, yI)))), qf(k));
    const uint32_t hi = (uint32_t)((uint64_t)(g ^ (g >> 63)) >> 32);
#if defined(__CUDA_ARCH__)
    const int lz = __clz((int)hi);
#else
    const int lz = hi ? __builtin_clz(hi) : 32;
#endif
    const int s = lz < 12 ? lz - 4 : 0;  // |g| < 1: lz >= 4 (32: k = 0)
    g <<= s;
    const int eF = f.r.e - 1023, x = 3 - eF - 2 * (i.e - 1023) - s + kx;  // (4 from the bracket, 2 of 2 t h)
    const Qf gf = qf(g), y2g = qf(qmul(qf(qmul(yF, yF)), gf));
    FxWall w;
    w.P = q_to_double(qmul(qf(Z3h), y2g), x - 1 - 2 * eF);
    w.R = q_to_double(qmul(qf(r3 + qhalf(r3)), y2g), x - 1 - 2 * eF + r3x);
    w.a = q_to_double(qmul(qf(qhalf(Z3h + rho3 + qhalf(rho3))), y2g), x - 2 * eF);
    w.c = q_to_double(qmul(qf(c4), gf), x);
    w.z = q_to_double(qmul(qf(z4), gf), x);
    return w;
}

// ---- matrix blocks ------------------------------------------------------------------------------
// G = A I + B d d^T, both times c
FLG_HD void fx_radial_block(const FxDir &g, const FxRadial &r, const FxConst &c, double *A, double *B) {
    const Qf cm = qf(c.m), y = qf(g.r.y);
    *A = q_to_double(qmul(qf(r.A), cm), r.x + c.x);
    *B = q_to_double(qmul(qf(qmul(qf(r.B), qf(qmul(y, y)))), cm), r.x + c.x - 2 * (g.r.e - 1023));
}
// the wall block from d0, d1 and: G_jk = a d_j d_k + c delta_jk, G_jz = d_j b1, G_zj = d_j b2, G_zz = z
// (j, k = x, y); t, h: the two heights, one of them times the constant
struct FxWallBlock {
    double a, b1, b2, c, z;
};
FLG_HD FxWallBlock fx_wall_block(double dm, double dp, double QF, double QI, double e, const FxConst &t, const FxConst &h) {
    const FxWall w = fx_wall(dm, dp, QF, QI, e, qmul(qf(t.m), qf(h.m)), t.x + h.x);
    const double Rd = w.R * dp;
    return {w.a, fma(w.P, dm, -Rd), fma(w.P, dm, Rd), w.c, w.z};
}

}  // namespace flg
