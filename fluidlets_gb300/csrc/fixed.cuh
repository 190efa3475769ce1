// fixed.cuh -- 60-bit fixed-point arithmetic for the FP64 pair kernels.
//
// GB300 issues one FP64 warp instruction per 64 clocks and scheduler (19 clocks per SM with all
// four busy), an integer multiply-add of 32 x 32 into 64 bits every 5 (1.3 per SM).  A product of
// two numbers of 60 fractional bits is three of those and two shifts, 4.2 clocks per SM, so
// whatever is bounded in a pair -- unit vectors, ratios, reciprocal square roots of a mantissa --
// is cheaper in fixed point than in FP64, at 2^-59 absolute error instead of 2^-54 relative.  The
// pair kernels (pair_fixed.cuh) form displacements and squared distances in FP64, which handles
// every range, move their mantissas here relative to the distance's exponent, and keep the
// exponents in integers.
//
// Q60: value = x 2^-60, |value| < 8; factors of a product must lie in [-2, 2).
#pragma once
#include <stdint.h>

#include <cmath>
#include <cstring>

#if defined(__CUDACC__)
#define FLG_HD __host__ __device__ __forceinline__
#else
#define FLG_HD inline
#endif

namespace flg {

typedef long long q60;
constexpr q60 kQ1 = 1ll << 60;  // 1.0

// a factor split into 30-bit limbs: x = h 2^30 + l (split once, used in several products)
struct Qf {
    int h, l;
};
FLG_HD Qf qf(q60 x) { return {(int)(x >> 30), (int)x & 0x3fffffff}; }
// a b, within 2^-60 of the product and without a bias: the constant in front of the shift is one
// half for rounding and one quarter for the mean of the low limbs' product that is left out (a sum
// over thousands of pairs would add a bias up, where it averages rounding errors)
FLG_HD q60 qmul(Qf a, Qf b) {
    const q60 t = (q60)a.l * b.h + ((q60)a.h * b.l + (3ll << 28));
    return (q60)a.h * b.h + (t >> 30);
}
// a b for a 30-bit b (Q30)
FLG_HD q60 qmul30(Qf a, int b) { return (q60)a.h * b + (((q60)a.l * b + (1ll << 29)) >> 30); }
// x / 2, rounded
FLG_HD q60 qhalf(q60 x) { return (x + 1) >> 1; }

FLG_HD uint64_t dbits(double x) {
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return u;
#endif
}
FLG_HD double bitsd(uint64_t u) {
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double x;
    std::memcpy(&x, &u, 8);
    return x;
#endif
}
FLG_HD int dexp(double x) { return (int)(dbits(x) >> 52) & 0x7ff; }  // biased exponent

// |x| 2^-(e - 1023) in Q60 for a normal x with biased exponent <= e (zero and denormals give at
// most 2^-60 too little of a unit that is not denormal)
FLG_HD q60 q_mag(double x, int e) {
    const uint64_t u = dbits(x);
    const int ex = (int)(u >> 52) & 0x7ff;
    const uint64_t m = ((u << 8) & 0x0fffffffffffff00ull) | 0x1000000000000000ull;
    const int sh = e - ex;
    return (q60)(m >> (sh < 63 ? sh : 63));
}
FLG_HD bool d_neg(double x) { return (int64_t)dbits(x) < 0; }
FLG_HD q60 q_sign(q60 m, bool neg) { return neg ? -m : m; }
// x 2^-(e - 1023), signed
FLG_HD q60 q_of(double x, int e) { return q_sign(q_mag(x, e), d_neg(x)); }

// seeds: the FP32 approximations as 30-bit integers (relative error below 2^-21)
FLG_HD int seed_rsqrt(float x) {  // x in [1, 4): 2^30 / sqrt(x)
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __float2int_rn(y * 1073741824.0f);
#else
    return (int)std::lrintf((1.0f / std::sqrt(x)) * 1073741824.0f);
#endif
}
FLG_HD int seed_rcp(float x) {  // x in [1, 2]: 2^30 / x
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __float2int_rn(y * 1073741824.0f);
#else
    return (int)std::lrintf((1.0f / x) * 1073741824.0f);
#endif
}
FLG_HD float bitsf(uint32_t u) {
#if defined(__CUDA_ARCH__)
    return __uint_as_float(u);
#else
    float x;
    std::memcpy(&x, &u, 4);
    return x;
#endif
}

// The square root of a positive normal Q: Q = q 2^(2 E), q in [1, 4), E = floor(exponent / 2).
struct QRsqrt {
    int e;    // E + 1023: q_mag(x, e) is |x| 2^-E for |x| <= sqrt(Q)
    q60 qh;   // q / 2
    q60 y;    // q^-1/2, in (1/2, 1]
};
// y0 (1 + c) with q y0^2 = 1 - 2 d, c = d + 3/2 d^2 (third order: d < 2^-20, so d^3 drops out)
FLG_HD QRsqrt q_rsqrt(double Q) {
    const uint64_t u = dbits(Q);
    const int ex = (int)(u >> 52) - 1023, odd = ex & 1;
    QRsqrt r;
    r.e = 1023 + ((ex - odd) >> 1);
    const uint64_t m = (u & 0x000fffffffffffffull) | 0x0010000000000000ull;
    r.qh = (q60)(m << (7 + odd));
    const int y0 = seed_rsqrt(bitsf(((uint32_t)(127 + odd) << 23) | ((uint32_t)(u >> 29) & 0x7fffffu)));
    const q60 d = (kQ1 >> 1) - qmul(qf(r.qh), qf((q60)y0 * y0));  // (1 - q y0^2) / 2
    const int ds = (int)(d >> 12);                               // Q48, below 2^29
    const q60 d2 = ((q60)ds * ds) >> 36;
    const q60 c = d + d2 + (d2 >> 1);
    r.y = ((q60)y0 << 30) + qmul30(qf(c), y0);
    return r;
}

// 1 / (1 + x) for x in [0, 1]: r0 (1 + c), (1 + x) r0 = 1 - d, c = d + d^2
FLG_HD q60 q_rcp1p(q60 x) {
    const q60 hp = (kQ1 + x) >> 1;  // (1 + x) / 2 in [1/2, 1]
    const int r0 = seed_rcp((float)(int)(hp >> 31) * (1.0f / 268435456.0f));
    const q60 d = kQ1 - 2 * qmul30(qf(hp), r0);
    const int ds = (int)(d >> 12);
    const q60 c = d + (((q60)ds * ds) >> 36);
    return ((q60)r0 << 30) + qmul30(qf(c), r0);
}

// x 2^p (x in Q60) as a double, rounded once (on the device by integer instructions, a tie away from zero: the FP64
// pipe, which converts, is what bounds the matrix kernels)
FLG_HD double q_to_double(q60 x, int p) {
    const int ex = p - 60;
#if defined(__CUDA_ARCH__)
    if (ex > 900 || ex < -900) return scalbn(__ll2double_rn(x), ex);
    const uint64_t s = (uint64_t)(x >> 63), m = ((uint64_t)x ^ s) - s;
    const int lz = __clzll((long long)m);
    const uint64_t n = m << (lz & 63);
    const uint64_t r = (n >> 11) + (n >> 10 & 1) + ((uint64_t)(uint32_t)(1085 - lz + ex) << 52);
    return bitsd(m == 0 ? 0 : r | (s & 0x8000000000000000ull));
#else
    const double d = (double)x;
    if (ex > 900 || ex < -900) return scalbn(d, ex);
    return x == 0 ? 0.0 : bitsd(dbits(d) + ((uint64_t)(int64_t)ex << 52));
#endif
}

}  // namespace flg
