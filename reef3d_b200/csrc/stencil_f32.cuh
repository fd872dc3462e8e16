// FP32 form of the level-set stencils.
//
// Uniform grids (the common case) use undivided differences: with
// q = (f[m+1]-f[m]) instead of (f[m+1]-f[m])/h, every smoothness indicator
// scales by h^2, so the WENO psi of the reference (1e-6,
// src/weno_nug_func.cpp:26) is rescaled to 1e-6*h^2 and the nonlinear
// weights come out identical in exact arithmetic; the reconstruction is
// divided by h once.  The classic Jiang-Peng coefficients used here are the
// values the reference's node tables take on a uniform grid (ideal weights
// 0.3/0.6/0.1, IS forms 10/3, 11/3, 4/3 of the q differences).
// Non-uniform grids use the reference's node tables in FP32 with divided
// differences.  The same templates run in FP64 for the interface band of
// the reinitialisation (see kernels_f32.cu).
#pragma once

#include "r3d_internal.h"

namespace r3d {
namespace f32 {

template <typename R>
__device__ __forceinline__ R rsqrt_r(R x) { return rsqrt(x); }
template <>
__device__ __forceinline__ float rsqrt_r<float>(float x) { return rsqrtf(x); }

// WENO5-HJ derivative on a uniform grid in FP64 (the interface band) from the
// undivided differences d1..d5 of the upwind set; eps = 1e-6*h^2.  Returns
// h * derivative.
__device__ __forceinline__ double weno5_uniform(bool plus, double d1, double d2, double d3, double d4, double d5,
                                                double eps) {
    // IS of the stencils (d3,d4,d5), (d2,d3,d4), (d1,d2,d3):
    // 10/3 a^2 + 11/3 ab + 4/3 b^2 with a, b the differences to the middle q
    const double a1 = d3 - d4, b1 = d5 - d4;
    const double a2 = d4 - d3, b2 = d2 - d3;
    const double a3 = d3 - d2, b3 = d1 - d2;
    const double k10 = 10.0 / 3.0, k11 = 11.0 / 3.0, k4 = 4.0 / 3.0;
    const double is1 = (k10 * a1 + k11 * b1) * a1 + k4 * b1 * b1;
    const double is2 = (k4 * a2 + (5.0 / 3.0) * b2) * a2 + k4 * b2 * b2;
    const double is3 = (k10 * a3 + k11 * b3) * a3 + k4 * b3 * b3;
    const double s1 = is1 + eps, s2 = is2 + eps, s3 = is3 + eps;
    const double r1 = 1.0 / s1, r2 = 1.0 / s2, r3 = 1.0 / s3;
    double c1, c2, c3;
    if (!plus) { c1 = 0.3; c2 = 0.6; c3 = 0.1; }
    else { c1 = 0.1; c2 = 0.6; c3 = 0.3; }
    const double al1 = c1 * r1 * r1, al2 = c2 * r2 * r2, al3 = c3 * r3 * r3;
    const double inv = 1.0 / (al1 + al2 + al3);
    double p1, p2, p3;
    if (!plus) {
        p1 = d4 + (1.0 / 3.0) * a1 - (1.0 / 6.0) * b1;
        p2 = d3 + (1.0 / 3.0) * a2 - (1.0 / 6.0) * b2;
        p3 = d2 + (1.0 / 3.0) * b3 + (11.0 / 6.0) * a3;
    } else {
        p1 = d4 + (11.0 / 6.0) * a1 + (1.0 / 3.0) * b1;
        p2 = d3 + (1.0 / 3.0) * b2 - (1.0 / 6.0) * a2;
        p3 = d2 + (1.0 / 3.0) * a3 - (1.0 / 6.0) * b3;
    }
    return (al1 * p1 + al2 * p2 + al3 * p3) * inv;
}

__device__ __forceinline__ float rcp_fast(float x) {  // 1 ulp
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// The reference's non-uniform form (tables, divided differences) in FP32,
// node tables of one (index, side) in the record W = Q0..Q5, C0..C2, S0..S8
// (8-byte aligned).  The weights c_r / s_r^2 over their sum are formed as
// c_r (m / s_r)^2 with m the smallest s_r, which stays in the FP32 range
// whatever the others are (an indicator that overflows has weight 0).  Four
// approximate reciprocals and no branch on the side, where four rounded ones,
// five quotients and both sides' code made a stretched 160 x 128 x 96 grid
// wait for them (stages of 40 / 66 us -> 37 / 48 us).
// The result is q3 plus the middle reconstruction's distance from it and the
// weighted distances of the others to the middle one: the weights' few ulp
// count against those alone (p1 w1 + p2 w2 + p3 w3 carries the sum's and the
// reciprocal's on the whole derivative), and a convection operator is 6.5e-8 to
// 7.2e-8 off the 64-bit one in the 2-norm (uniform grids 5.5e-8 to 6.8e-8), where
// the form with rounded reciprocals and quotients was 9.3e-8 to 1.0e-7 (8.0e-8 to
// 9.5e-8) off.
// MASKS: the weight of stencil (q3,q4,q5) / (q2,q3,q4) / (q1,q2,q3) is 0 where
// zero1..zero3 (the X45 = 6 masked differences; at least one stays on), and
// the unscaled c_r / s_r^2 leave the FP32 range (no finite result) where the
// caller is to evaluate in FP64.
template <bool MASKS = false>
__device__ __forceinline__ float weno5_tables(const float* __restrict__ W, bool plus, float q1, float q2, float q3,
                                              float q4, float q5, bool zero1 = false, bool zero2 = false,
                                              bool zero3 = false) {
    float w[18];
#pragma unroll
    for (int m = 0; m < 9; ++m) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(W) + m);
        w[2 * m] = v.x;
        w[2 * m + 1] = v.y;
    }
    const float *Q = w, *C = w + 6, *S = w + 9;
    const float dq12 = q1 - q2, dq23 = q2 - q3, dq34 = q3 - q4, dq54 = q5 - q4;
    const float s1 = (S[0] * dq54 + S[1] * dq34) * dq54 + S[2] * dq34 * dq34 + 1.0e-6f;
    const float s2 = (S[3] * dq23 - S[4] * dq34) * dq23 + S[5] * dq34 * dq34 + 1.0e-6f;
    const float s3 = (S[6] * dq12 - S[7] * dq23) * dq12 + S[8] * dq23 * dq23 + 1.0e-6f;
    float n1, n2, n3;
    if (MASKS) {
        const float u1 = __frcp_rn(s1), u2 = __frcp_rn(s2), u3 = __frcp_rn(s3);
        n1 = zero1 ? 0.0f : C[0] * u1 * u1;
        n2 = zero2 ? 0.0f : C[1] * u2 * u2;
        n3 = zero3 ? 0.0f : C[2] * u3 * u3;
    } else {
        const float m = fminf(s1, fminf(s2, s3));
        const float u1 = m * rcp_fast(s1), u2 = m * rcp_fast(s2), u3 = m * rcp_fast(s3);
        n1 = C[0] * u1 * u1;
        n2 = C[1] * u2 * u2;
        n3 = C[2] * u3 * u3;
    }
    const float t1 = Q[1] * dq54;
    const float x2 = plus ? dq23 : -dq34, y2 = plus ? -dq34 : dq23;
    const float x3 = plus ? -dq23 : dq12, y3 = plus ? dq12 : -dq23;
    const float t3 = Q[5] * y3;
    const float r1 = Q[0] * dq34 + (plus ? t1 : -t1);
    const float r2 = Q[2] * x2 - Q[3] * y2;
    const float r3 = Q[4] * x3 + (plus ? -t3 : t3);
    if (MASKS) return (n1 * (q4 + r1) + n2 * (q3 + r2) + n3 * (q2 + r3)) * __frcp_rn(n1 + n2 + n3);
    return q3 + (r2 + (n1 * (r1 - (dq34 + r2)) + n3 * (r3 + (dq23 - r2))) * rcp_fast(n1 + n2 + n3));
}

// The uniform form in FP32 from the upwind set d1..d5 (the plus side passes
// the mirrored set), weights as in weno5_tables; eps = 1e-6 h^2.  Returns h
// times the derivative.
__device__ __forceinline__ float weno5_mirrored(float d1, float d2, float d3, float d4, float d5, float eps) {
    const float a1 = d3 - d4, b1 = d5 - d4, b2 = d2 - d3, b3 = d1 - d2;
    const float k10 = 10.0f / 3.0f, k11 = 11.0f / 3.0f, k5 = 5.0f / 3.0f, k4 = 4.0f / 3.0f;
    const float s1 = (k10 * a1 + k11 * b1) * a1 + (k4 * b1 * b1 + eps);
    const float s2 = (k4 * a1 - k5 * b2) * a1 + (k4 * b2 * b2 + eps);
    const float s3 = (k10 * b2 - k11 * b3) * b2 + (k4 * b3 * b3 + eps);
    const float m = fminf(s1, fminf(s2, s3));
    const float u1 = m * rcp_fast(s1), u2 = m * rcp_fast(s2), u3 = m * rcp_fast(s3);
    const float n1 = 0.3f * u1 * u1, n2 = 0.6f * u2 * u2, n3 = 0.1f * u3 * u3;
    // the reconstructions as d3 + m2 (the middle one) and differences to it
    const float m2 = -(1.0f / 3.0f) * a1 - (1.0f / 6.0f) * b2;
    const float e1 = -(2.0f / 3.0f) * a1 - (1.0f / 6.0f) * b1 - m2;
    const float e3 = (1.0f / 3.0f) * b3 - (5.0f / 6.0f) * b2 - m2;
    return d3 + (m2 + (n1 * e1 + n3 * e3) * rcp_fast(n1 + n2 + n3));
}

// Derivative along an axis of a uniform grid from the 7 values fv[0..6] =
// f[-3..3] around the cell (already divided by h).
__device__ __forceinline__ double deriv_uniform(const double* fv, bool plus, double rh, double eps) {
    if (!plus)
        return rh * weno5_uniform(false, fv[1] - fv[0], fv[2] - fv[1], fv[3] - fv[2], fv[4] - fv[3], fv[5] - fv[4],
                                  eps);
    return rh * weno5_uniform(true, fv[2] - fv[1], fv[3] - fv[2], fv[4] - fv[3], fv[5] - fv[4], fv[6] - fv[5], eps);
}

__device__ __forceinline__ float deriv_uniform(const float* fv, bool plus, float rh, float eps) {
    float D[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) D[m] = fv[m + 1] - fv[m];
    return rh * weno5_mirrored(plus ? D[5] : D[0], plus ? D[4] : D[1], plus ? D[3] : D[2], plus ? D[2] : D[3],
                               plus ? D[1] : D[4], eps);
}

// dpr: the (DXP, 1/DXP) pairs, wt: the node records, of the axis.
__device__ __forceinline__ float deriv_tables(const float* fv, bool plus, const float* __restrict__ dpr,
                                              const float* __restrict__ wt, int t) {
    float q[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) q[m] = (fv[m + 1] - fv[m]) * __ldg(dpr + 2 * (t + m - 3) + 1);
    return weno5_tables(wt + 18 * (2 * t + (plus ? 1 : 0)), plus, plus ? q[1] : q[0], plus ? q[2] : q[1],
                        plus ? q[3] : q[2], plus ? q[4] : q[3], plus ? q[5] : q[4]);
}

// Reinitialisation right-hand side from the axis stencils (7 values per
// axis, centre at [3]); the Godunov selection and smoothed sign of
// src/reinidisc_f.cpp:58-127 on a uniform grid.  rh[a] = 1/h_a,
// hh[a] = h_a^2, eps = the reference's WENO psi (1e-6).
template <typename R, bool TWO_D>
__device__ __forceinline__ R reini_rhs_uniform(const R* fx, const R* fy, const R* fz, const R* rh, const R* hh,
                                               R eps, R deltax) {
    const R lsv = fx[3];
    const R lsSig = (fabs((double)lsv) < 1.0e-8) ? R(1) : (lsv > R(0) ? R(1) : R(-1));
    R g[3] = {R(0), R(0), R(0)};
    const R* fa[3] = {fx, fy, fz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (TWO_D && a == 1) continue;
        const R* f = fa[a];
        const R xmin = (lsv - f[2]) * rh[a];
        const R xplus = (f[4] - lsv) * rh[a];
        // minus side, plus side, or neither; one evaluation for both sides
        const bool c1 = xmin * lsSig > R(0) && xplus * lsSig > -xmin * lsSig;
        const bool c2 = xplus * lsSig < R(0) && xmin * lsSig < -xplus * lsSig;
        const R d = deriv_uniform(f, c2, rh[a], eps * hh[a]);
        g[a] = c1 || c2 ? d : R(0);
    }
    const R dnorm = sqrt(g[0] * g[0] + g[1] * g[1] + g[2] * g[2]);
    R sign = lsv * rsqrt_r(lsv * lsv + dnorm * dnorm * deltax * deltax);
    if (sign != sign) sign = R(1);
    return -(sign * dnorm - sign);
}

}  // namespace f32
}  // namespace r3d
