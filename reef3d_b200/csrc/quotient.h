// FP64 quotients rounded to nearest from bounds of the reciprocals, for several
// divisions that share their divisors.  Plain arithmetic (fma and products), so
// that the host can check it.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define R3D_HD __host__ __device__ __forceinline__
#else
#define R3D_HD inline
#endif

namespace r3d {
namespace f64 {

// A lower bound of 1/b, 2^-48 to 2^-35.9 below it, from y, an approximation with
// |1 - b y| <= 2^-18: one Newton step, y (1 + e) = (1 - e^2)/b, never exceeds
// 1/b, and is pushed 2^-48 further down (past its own rounding, 2^-53).  The
// product of two such bounds is one of 1/(b c), down to 2^-34.9.
R3D_HD double reciprocal_below(double b, double y) { return fma(y, fma(-b, y, 1.0 - 0x1p-48), y); }

R3D_HD uint32_t low_word(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return (uint32_t)u;
#endif
}

// a / b rounded to nearest, or `apart` made nonzero; y from reciprocal_below (or
// a product of two).  With q near a/b and the remainder r = a - b q (rounded, a
// relative 2^-53), a/b = q + r/b lies between q + r y and q + r y (1 + 2^-34).
// Rounding is monotone, so where the two round to the same double, a/b does
// too; where they differ (a/b within 2^-15 of an ulp of the middle of two
// doubles: the bracket's width times q's distance) the caller divides.  For
// a and quotients within 2^+-960.
R3D_HD double bracket_div(double a, double b, double y, uint32_t& apart) {
    const double q = a * y;
    const double r = fma(-b, q, a);
    const double l = fma(r, y, q), h = fma(fma(r, 0x1p-34, r), y, q);
    apart |= low_word(l) ^ low_word(h);
    return l;
}

}  // namespace f64
}  // namespace r3d
