// Exactly rounded reciprocals and quotients without a division's range branch,
// for chains in which several values are divided by one.
#pragma once
#include <cuda_runtime.h>

namespace verb {
namespace {

// RN(1 / x) for 2^-1021 <= |x| < 2^1022, where x, 1/x and the steps stay normal:
// Newton steps from the hardware's approximation, the last one correcting by the
// exact residual, which rounds correctly except where the significand of x is all
// ones (Markstein, IBM J. Res. Dev. 34, 1990); there 1/x lies just above the
// midpoint of a power of two and its successor and rounds to the successor.
__device__ __forceinline__ double recip(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#pragma unroll
    for (int i = 0; i < 4; i++) y = fma(y, fma(-x, y, 1.0), y);
    const long long ones = 0xfffffffffffffLL;
    const bool all = (__double_as_longlong(x) & ones) == ones;
    return all ? __longlong_as_double(__double_as_longlong(y) | 1) : y;
}

// a / b rounded to nearest with y = RN(1/b) (one correction of the product by
// its residual, Markstein) for |a|, |b| in [2^-400, 2^400), where neither the
// quotient nor the residual leaves the normal range; others are divided.
__device__ __forceinline__ double div_by(double a, double b, double y)
{
    const double q = a * y;
    const unsigned ea = ((unsigned)__double2hiint(a) & 0x7fffffffu) - 0x26f00000u;
    const unsigned eb = ((unsigned)__double2hiint(b) & 0x7fffffffu) - 0x26f00000u;
    if (eb < 0x32000000u) {
        if (ea < 0x32000000u) return fma(fma(-q, b, a), y, q);
        if (a == 0.0) return q;
    }
    return a / b;
}

}  // namespace
}  // namespace verb
