// slices.cuh -- FP64 numbers as eight 8-bit integer digits relative to a common exponent, the
// operand format of the FP64-accurate tensor-core product (slice_gemm.cu).
//
// A row (or column) of FP64 values with |x| < 2^e is written as
//     x = 2^(e - 62) sum_{k=0..7} d_k 256^(7-k),   d_k integer in [-128, 127],
// i.e. as a 62-bit fixed-point number in balanced base-256 digits: exact for values within a
// factor 2^9 of 2^e, rounded to 2^(e - 63) below.  A digit is exact in BF16 (8 significant
// bits), a product of two digits is an integer of at most 2^14, and 64 x 8 such products sum to
// at most 2^23, which FP32 accumulates exactly.
//
// What that costs a dot product of a row and a column depends on where their large values meet: its
// error is about 2^-59 of 2^(ea + eb), which is small beside the FP64 rounding errors of a term that
// is large in both and not small at all where every product lies far below the two maxima (rows
// of different units among the 64 pivots).  The masks of a row or column say which of its 64 values
// reach 2^(e - 1 - near), and which are not zero; slice_gemm.cu recomputes in FP64 what the masks of a row
// and a column leave open.
#pragma once
#include <stdint.h>

namespace flg {

constexpr int kSlices = 8;            // digits per value
constexpr int kSliceK = 64;           // depth of one operand block: 64 BF16 = 128 bytes
constexpr int kSliceNonFinite = 1 << 20;  // exponent of a row or column that holds an Inf or NaN
typedef uint4 SliceMask;              // near (x, y), non-zero (z, w); value k: bit k / 2 of the first word, odd k of the second

// biased exponent of x, 1 for zero and denormals (they scale like the smallest normals)
__device__ __forceinline__ int slice_exponent(double x) {
    const int ex = (__double2hiint(x) >> 20) & 0x7ff;
    return ex ? ex : 1;
}
// the common exponent e (|x| < 2^e) from the largest biased exponent of the row
__device__ __forceinline__ int slice_scale(int exmax) { return exmax == 0x7ff ? kSliceNonFinite : exmax - 1022; }

// whether x counts as near the maximum of its row or column
__device__ __forceinline__ bool slice_near(double x, int exmax, int near) {
    return exmax == 0x7ff || slice_exponent(x) >= exmax - near;
}
// the masks' range for n unknowns: products of near values reach 2^(ea + eb - (2 near + 2)), and 2 near + 2 is at
// most log2 n + 4 (slice_gemm.cu)
inline int slice_near_range(int64_t n) {
    int lg = 0;
    while (n >> (lg + 1)) lg++;
    return (lg + 2) / 2;
}

// the eight digits of x relative to the row's largest biased exponent, biased by 128: digit k is
// byte 7 - k of the result minus 128 (zero digits for a row with non-finite entries)
__device__ __forceinline__ uint64_t slice_digits(double x, int exmax) {
    const uint64_t bias = 0x8080808080808080ull;
    if (exmax == 0x7ff) return bias;
    const uint64_t u = (uint64_t)__double_as_longlong(x);
    const int ex = (int)(u >> 52) & 0x7ff;
    const uint64_t mant = (u & 0xfffffffffffffull) | (ex ? 0x10000000000000ull : 0ull);
    const int sh = 9 - (exmax - (ex ? ex : 1));
    uint64_t F;
    if (sh >= 0) F = mant << sh;
    else if (sh > -54) F = (mant + (1ull << (-sh - 1))) >> -sh;
    else F = 0;
    return ((int64_t)u < 0 ? 0ull - F : F) + bias;
}

// digit k of a biased digit word as the upper half of an FP32 number, i.e. its BF16 bits << 16
__device__ __forceinline__ uint32_t slice_bf16_hi(uint64_t w, int k) {
    const uint32_t b = (uint32_t)(w >> (8 * (7 - k))) & 0xffu;
    return __float_as_uint(__uint_as_float(0x4b000000u | b) - 8388736.0f);  // 2^23 + b - (2^23 + 128)
}

}  // namespace flg
