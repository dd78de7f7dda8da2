// The face polynomial of Convection_1D_ULTIMATE_QUICKEST6 (QUICKEST6.cpp:
// 162-241) with its Courant factors, shared by the line-job kernels
// (convection.cu) and the two-stage kernel (convection_staged.cu).  Compiled
// without contraction the operations are the reference's, one by one.
#pragma once
#include <cuda_runtime.h>

namespace verb {
namespace {

// Courant-number factors of the face polynomial (QUICKEST6.cpp:209-238); they
// depend only on the face Courant number.
struct FaceCoef {
    double k3, c6, k5, k7, k9;
};

// The face value with the Courant factors supplied: the reference's operations
// in its order.
__device__ __forceinline__ double quickest_face_k(double U1, double U2, double U3, double U4,
                                                  double C, double D1, double D2v, double D3v,
                                                  double D4v, double D5v, double cr,
                                                  const FaceCoef& k)
{
    const double ca = fabs(cr);
    double f = 0.5 * (C + D1);
    const double d1 = C - D1;
    f += 0.5 * ca * d1;
    const double D2 = (U1 - C - D1 + D2v) / 2;
    const double d3 = U1 - 3 * C + 3 * D1 - D2v;
    f += k.k3 * (D2 + ca / 4 * d3);
    const double D4 = (U2 - 3 * U1 + 2 * C + 2 * D1 - 3 * D2v + D3v) / 2;
    const double d5 = U2 - 5 * U1 + 10 * C - 10 * D1 + 5 * D2v - D3v;
    f += k.k5 * (D4 + k.c6 * d5);
    const double D6 = (U3 - 5 * U2 + 9 * U1 - 5 * C - 5 * D1 + 9 * D2v - 5 * D3v + D4v) / 2;
    const double d7 = U3 - 7 * U2 + 21 * U1 - 35 * C + 35 * D1 - 21 * D2v + 7 * D3v - D4v;
    f += k.k7 * (D6 + ca / 8 * d7);
    const double D8 = (U4 - 7 * U3 + 20 * U2 - 28 * U1 + 14 * C + 14 * D1 - 28 * D2v + 20 * D3v -
                       7 * D4v + D5v) /
                      2;
    const double d9 = U4 - 9 * U3 + 36 * U2 - 84 * U1 + 126 * C - 126 * D1 + 84 * D2v - 36 * D3v +
                      9 * D4v - D5v;
    f += k.k9 * (D8 + d9 / 2);
    return f;
}

// a / b rounded to nearest, for the constants b = 6, 120, 5040 and 362880 with
// y = RN(1/b) (Markstein's correction step: P. Markstein, IBM J. Res. Dev.
// 34(1), 1990).  q = RN(a*y) is within 1.5 ulp of a/b, so the residual a - b*q
// is a representable number (at most 6B units of 2^(e_b+e_q-1), B <= 2835 the
// odd part of b) and the fused multiply-add returns it exactly.  q + r*y then
// differs from a/b by |r|*|y - 1/b| < 1.5*2^-53 ulp, whereas a/b lies at
// least ulp/(2B) away from every rounding midpoint (b's odd part B >= 3 makes
// a midpoint times b need more than 53 significant bits), so a single
// rounding of q + r*y gives RN(a/b).  A zero residual returns q, which keeps
// the sign that division gives to a zero quotient.
__device__ __forceinline__ double div_const(double a, double b, double y)
{
    const double q = __dmul_rn(a, y);
    const double r = __fma_rn(-q, b, a);
    return r == 0.0 ? q : __fma_rn(r, y, q);
}

// The same for a dividend that is never -0 (then a zero residual needs no
// special case: q + 0*y = q for every q but -0).
__device__ __forceinline__ double div_const_nz(double a, double b, double y)
{
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

// Courant factors of the face polynomial (QUICKEST6.cpp:209-238), with
// exactly rounded divisions by the constant denominators.
__device__ __forceinline__ FaceCoef face_coef_exact(double cr)
{
    const double cs = cr * cr;
    const double ca = fabs(cr);
    const double t1 = cs - 1;
    const double p2 = t1 * (cs - 4);
    const double p3 = p2 * (cs - 9);
    const double p4 = p3 * (cs - 16);
    // t1 = cs - 1 and ca = |cr| are never -0, nor is p3 = p2*(cs-9) (p2 = -0
    // only when cs = 1, and then p3 = +0); p2 and p4 are -0 when |cr| = 1
    FaceCoef k;
#ifdef VERB_BUILD_CONV_FMA
    // contracted form: a product with the rounded reciprocal (within an ulp
    // of the quotient) instead of the exactly rounded division
    k.k3 = t1 * (1.0 / 6.0);
    k.c6 = ca * (1.0 / 6.0);
    k.k5 = p2 * (1.0 / 120.0);
    k.k7 = p3 * (1.0 / 5040.0);
    k.k9 = p4 * (1.0 / 362880.0);
#else
    k.k3 = div_const_nz(t1, 6.0, 1.0 / 6.0);
    k.c6 = div_const_nz(ca, 6.0, 1.0 / 6.0);
    k.k5 = div_const(p2, 120.0, 1.0 / 120.0);
    k.k7 = div_const_nz(p3, 5040.0, 1.0 / 5040.0);
    k.k9 = div_const(p4, 362880.0, 1.0 / 362880.0);
#endif
    return k;
}

}  // namespace
}  // namespace verb
