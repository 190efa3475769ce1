// pair_fixed.cuh -- the FP64 pair kernels in 60-bit fixed point (fixed.cuh).
//
// The same formulas as pair_math.cuh's, written in bounded quantities.  With Q = |d|^2 + e^2 =
// q 2^(2E), y = q^-1/2, the unit vector n = d / sqrt(Q) and w = e / sqrt(Q):
//   Stokeslet     8 pi u = s [(1 + w^2) f + (f.n) n],                       s = y 2^-E
//   Brinkmanlet   4 pi u = s [(f1 + w^2 f2) f + f2 (f.n) n]                 below z = 1/2 (series), and
//                        = s^3 / alpha^2 [(F1 + w^2 F2) f + F2 (f.n) n],    F = z^2 f, above:
//     F1 = E (1 + z + z^2) - 1, F2 = 3 - E (3 + 3 z + z^2), E = e^-z from 2^-n 2^(-i/64) e^-x with a table
//     (P. T. P. Tang, "Table-driven implementation of the exponential function in IEEE
//     floating-point arithmetic", ACM TOMS 15, 1989)
//   wall          8 pi u = 2 t h sF s^2 [...] with rho = s / sF <= 1, nI = dp s and the bracket
//     c f_j + n_j (Z3 (f.n) - 3 rho^2 B)           (j = x, y),  c = Z1 + w^2 Z3 - rho + 3 w^2 rho^3
//     c' f_z + n_z Z3 (f.n) - 3 rho nI B,                       c' = Z1 + w^2 Z3 - rho - 3 w^2 rho^3
//     Z1 = 2 / (1 + rho), Z3 = Z1 (1 + rho + rho^2) = 2 + ... , B = nI f_z - rho (n_x f_x + n_y f_y)
//   (the bracket is the image form of pair_math.cuh divided by sF^3 rho^2, which keeps its
//   precision where the wall is far: rho -> 0).
// Displacements and Q stay in FP64 (their rounding is the FP64 kernel's own); everything after them
// is an integer of 2^-59 absolute error in quantities of order one, where an FP64 chain of the
// same length has several 2^-54 relative ones.  Pairs outside the ranges where this holds (Q
// not a normal number far from the limits, strengths that are not finite, targets and sources on
// opposite sides of the wall) go to the FP64 functions, pair by pair.
#pragma once
#include "fixed.cuh"

namespace flg {

// exponents of Q that the fixed-point path takes: every exponent sum stays far inside the range
constexpr int kQExpMin = 1023 - 1000, kQExpMax = 1023 + 1000;
FLG_HD bool q_in_range(double Q) {
    const int ex = (int)(dbits(Q) >> 52);  // (a sign bit makes it too large)
    return ex >= kQExpMin && ex <= kQExpMax;
}

// strengths of one source, f = F 2^e with the largest |F_k| in [1/4, 1/2); e = kFxBad: not finite
constexpr int kFxBad = 1 << 28, kFxZero = -(1 << 20);
FLG_HD int fx_strength(const double *f, int n, q60 *F) {
    int em = 0;
    for (int k = 0; k < n; k++) em = dexp(f[k]) > em ? dexp(f[k]) : em;
    if (em == 0x7ff) return kFxBad;
    for (int k = 0; k < n; k++) F[k] = q_of(f[k], em) >> 2;  // |f| 2^-em < 2: a quarter of it below 1/2
    return em < 64 ? (em == 0 ? kFxZero : kFxBad) : em - 1023 + 2;
}

// what the pair kernels give: the coefficients of u = (A f + B (f.n) n) 2^x for a radial kernel
struct FxRadial {
    q60 A, B;  // A in [-1.8, 1.8], B in [0, 1.6]
    int x;
};
struct FxDir {  // unit vector and w^2, with the root
    q60 n[3], w2;
    QRsqrt r;
};
FLG_HD FxDir fx_dir(double d0, double d1, double d2, double Q, double e) {
    FxDir g;
    g.r = q_rsqrt(Q);
    const Qf y = qf(g.r.y);
    g.n[0] = q_sign(qmul(qf(q_mag(d0, g.r.e)), y), d_neg(d0));
    g.n[1] = q_sign(qmul(qf(q_mag(d1, g.r.e)), y), d_neg(d1));
    g.n[2] = q_sign(qmul(qf(q_mag(d2, g.r.e)), y), d_neg(d2));
    const Qf w = qf(qmul(qf(q_mag(e, g.r.e)), y));
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

// u / 2^x for strengths F; |u| < 2
FLG_HD void fx_radial_apply(const FxDir &g, const FxRadial &r, const q60 *F, q60 *u) {
    const Qf n0 = qf(g.n[0]), n1 = qf(g.n[1]), n2 = qf(g.n[2]), f0 = qf(F[0]), f1 = qf(F[1]), f2 = qf(F[2]);
    const q60 t = qmul(f0, n0) + qmul(f1, n1) + qmul(f2, n2);
    const Qf b = qf(qmul(qf(t), qf(r.B))), A = qf(r.A);
    u[0] = qmul(A, f0) + qmul(b, n0);
    u[1] = qmul(A, f1) + qmul(b, n1);
    u[2] = qmul(A, f2) + qmul(b, n2);
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

// the two parts of one real strength vector: ur = (Ar F + Br t n), ui = (Ai F + Bi t n), t = F.n
FLG_HD void fx_radial_apply_c(const FxDir &g, const FxRadialC &r, const q60 *F, q60 *ur, q60 *ui) {
    const Qf n0 = qf(g.n[0]), n1 = qf(g.n[1]), n2 = qf(g.n[2]), f0 = qf(F[0]), f1 = qf(F[1]), f2 = qf(F[2]);
    const Qf t = qf(qmul(f0, n0) + qmul(f1, n1) + qmul(f2, n2));
    const Qf br = qf(qmul(t, qf(r.Br))), bi = qf(qmul(t, qf(r.Bi))), Ar = qf(r.Ar), Ai = qf(r.Ai);
    ur[0] = qmul(Ar, f0) + qmul(br, n0);
    ur[1] = qmul(Ar, f1) + qmul(br, n1);
    ur[2] = qmul(Ar, f2) + qmul(br, n2);
    ui[0] = qmul(Ai, f0) + qmul(bi, n0);
    ui[1] = qmul(Ai, f1) + qmul(bi, n1);
    ui[2] = qmul(Ai, f2) + qmul(bi, n2);
}

// wall: everything that does not depend on the strengths
struct FxWall {
    q60 nx, ny, nm, nI, rho, rho2, Z3h, cq, czq, g, yF;
    q60 r3;  // rho^3 = r3 2^r3x, r3 in [1/8, 1): with its relative precision where rho is small
    int r3x;
    int eF;  // sF = yF 2^-eF
    int x;  // bracket / 8 . g . 2^x, without the factor t h
};
FLG_HD FxWall fx_wall(double d0, double d1, double dm, double dp, double QF, double QI, double e) {
    const FxDir f = fx_dir(d0, d1, dm, QF, e);
    const QRsqrt i = q_rsqrt(QI);
    const Qf yI = qf(i.y);
    FxWall w;
    w.nx = f.n[0], w.ny = f.n[1], w.nm = f.n[2];
    w.nI = q_sign(qmul(qf(q_mag(dp, i.e)), yI), d_neg(dp));
    // rho = (yI / yF) 2^(EF - EI), 1 / yF = q yF
    const q60 half = qmul(yI, qf(qmul(qf(f.r.qh), qf(f.r.y))));
    w.rho = q_shift(half << 1, i.e - f.r.e);
    if (w.rho > kQ1) w.rho = kQ1;
    const int low = half < kQ1 / 2;  // (1/4 < half < 1)
    const Qf rm = qf(half << low);
    w.r3 = qmul(rm, qf(qmul(rm, rm)));
    w.r3x = 3 * (1 - low - (i.e - f.r.e));
    const Qf rho = qf(w.rho);
    w.rho2 = qmul(rho, rho);
    const q60 Z1h = q_rcp1p(w.rho);  // Z1 / 2
    w.Z3h = kQ1 + qmul(qf(w.rho2), qf(Z1h));  // Z3 / 2 = 1 + rho^2 / (1 + rho)
    const q60 w2r3 = qmul(qf(f.w2), qf(qmul(qf(w.rho2), rho)));
    const q60 base = Z1h + qmul(qf(f.w2), qf(w.Z3h)) - qhalf(w.rho), i3 = w2r3 + qhalf(w2r3);
    w.cq = qhalf(base + i3), w.czq = qhalf(base - i3);  // c / 4, c' / 4
    w.g = qmul(qf(f.r.y), qf(qmul(yI, yI)));
    w.yF = f.r.y, w.eF = f.r.e - 1023;
    w.x = 4 - w.eF - 2 * (i.e - 1023);  // 8 from the bracket, 2 of 2 t h
    return w;
}
// the exponent of u 2^x is returned: the bracket cancels near the wall and for far images, so it is
// scaled up to [1/2, 1) before its last product
FLG_HD int fx_wall_apply(const FxWall &w, const q60 *F, q60 *u) {
    const Qf nx = qf(w.nx), ny = qf(w.ny), nm = qf(w.nm), nI = qf(w.nI), f0 = qf(F[0]), f1 = qf(F[1]), f2 = qf(F[2]);
    const q60 D = qmul(f0, nx) + qmul(f1, ny);
    const Qf B = qf(qmul(nI, f2) - qmul(qf(w.rho), qf(D)));
    const q60 t1 = qmul(qf(w.Z3h), qf(D + qmul(f2, nm)));  // Z3 (f.n) / 2
    const q60 r2B = qmul(qf(w.rho2), B), zB = qmul(qf(w.rho), qf(qmul(nI, B)));
    const Qf b = qf(qhalf(t1 - r2B - qhalf(r2B))), cq = qf(w.cq), g = qf(w.g);
    const q60 ux = qmul(cq, f0) + qmul(b, nx), uy = qmul(cq, f1) + qmul(b, ny);
    const q60 uz = qmul(qf(w.czq), f2) + qhalf(qmul(nm, qf(t1)) - zB - qhalf(zB));
    const uint64_t m = (uint64_t)((ux ^ (ux >> 63)) | (uy ^ (uy >> 63)) | (uz ^ (uz >> 63)));
#if defined(__CUDA_ARCH__)
    const int lz = __clz((int)(m >> 32));
#else
    const int lz = (m >> 32) ? __builtin_clz((unsigned)(m >> 32)) : 32;
#endif
    // |bracket| / 4 < 2.4: lz >= 2; one shift left of lz - 3 after the shift right that makes room
    const int s = lz < 5 ? 0 : lz - 5;
    u[0] = qmul(qf(qhalf(ux << s)), g);
    u[1] = qmul(qf(qhalf(uy << s)), g);
    u[2] = qmul(qf(qhalf(uz << s)), g);
    return w.x - s;
}

// ---- matrix blocks ------------------------------------------------------------------------------
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

// G = A I + B d d^T, both times c
FLG_HD void fx_radial_block(const FxDir &g, const FxRadial &r, const FxConst &c, double *A, double *B) {
    const Qf cm = qf(c.m), y = qf(g.r.y);
    *A = q_to_double(qmul(qf(r.A), cm), r.x + c.x);
    *B = q_to_double(qmul(qf(qmul(qf(r.B), qf(qmul(y, y)))), cm), r.x + c.x - 2 * (g.r.e - 1023));
}
// the wall block from d0, d1 and: G_jk = a d_j d_k + c delta_jk, G_jz = d_j b1, G_zj = d_j b2, G_zz = z
// (j, k = x, y); t, h: the two heights, one of them times the constant.  With P = Z3 k, R = 3 rho^3 k of
// the common factor k, a = P + R, b1 = P dm - R dp, b2 = P dm + R dp in FP64: beside the distance dm and dp may be small,
// and b1 and b2 keep their precision to 2^-53 of their own terms.  (As fixed-point n_z and n_I to 2^-60 of the
// distance, at heights of 1e-6 of it b1 and b2 were exact to 5e-13.)
struct FxWallBlock {
    double a, b1, b2, c, z;
};
FLG_HD FxWallBlock fx_wall_block(double d0, double d1, double dm, double dp, double QF, double QI, double e,
                                 const FxConst &t, const FxConst &h) {
    const FxWall w = fx_wall(d0, d1, dm, dp, QF, QI, e);
    // g t h, scaled up to [1/2, 1)
    q60 k = qmul(qf(w.g), qf(qmul(qf(t.m), qf(h.m))));
    const uint32_t hi = (uint32_t)((uint64_t)(k ^ (k >> 63)) >> 32);
#if defined(__CUDA_ARCH__)
    const int lz = __clz((int)hi);
#else
    const int lz = hi ? __builtin_clz(hi) : 32;
#endif
    const int s = lz < 12 ? lz - 4 : 0;  // |k| < 1: lz >= 4 (0: t = 0)
    k <<= s;
    const Qf kf = qf(k), yf = qf(w.yF), nm = qf(w.nm), nI = qf(w.nI);
    const q60 rn2 = qmul(qf(w.rho), qf(qmul(nI, nI)));
    const q60 z4 = w.czq + qhalf(qmul(nm, qf(qmul(qf(w.Z3h), nm))) - rn2 - qhalf(rn2));
    const int x = w.x - 1 - s + t.x + h.x;  // (the bracket over 4 here, over 8 in w.x)
    const Qf y2k = qf(qmul(qf(qmul(yf, yf)), kf));
    const double P = q_to_double(qmul(qf(w.Z3h), y2k), x - 1 - 2 * w.eF);
    const double R = q_to_double(qmul(qf(w.r3 + qhalf(w.r3)), y2k), x - 1 - 2 * w.eF + w.r3x), Rd = R * dp;
    FxWallBlock b;
    b.a = P + R;
    b.b1 = fma(P, dm, -Rd);
    b.b2 = fma(P, dm, Rd);
    b.c = q_to_double(qmul(qf(w.cq), kf), x);
    b.z = q_to_double(qmul(qf(z4), kf), x);
    return b;
}

// Sums of up to 16 terms u 2^x with |u| < 2: 64-bit integers of 57 fractional bits (a term is
// rounded to 2^-58 of its unit, the sum stays below 2^62) relative to the largest exponent so far,
// which outlives the 16 terms.
constexpr int kFxSeg = 16;
template <int NC>
struct FxAcc {
    q60 a[NC];
    int x;
    FLG_HD void init() {
        clear();
        x = -(1 << 24);
    }
    FLG_HD void clear() {
        for (int k = 0; k < NC; k++) a[k] = 0;
    }
    // makes room for a term of exponent xt (rare once the first few pairs have passed)
    FLG_HD void scale(int xt) {
        if (xt > x) {
            const int s = xt - x < 63 ? xt - x : 63;
            for (int k = 0; k < NC; k++) a[k] = qshr(a[k], s);
            x = xt;
        }
    }
    // term u[0..3) of exponent xt at component c0 of the sum
    FLG_HD void add(int c0, const q60 *u, int xt) {
        const int s = x - xt + 3 < 63 ? x - xt + 3 : 63;
        for (int k = 0; k < 3; k++) a[c0 + k] += qshr(u[k], s);
    }
    FLG_HD double value(int k) const { return q_to_double(a[k], x + 3); }
};

}  // namespace flg
