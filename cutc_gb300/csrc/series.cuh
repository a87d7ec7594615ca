// FP64 1/sqrt(x) and 1/x from FP32 seeds, by one step of third order: with the seed's residual
// e = 1 - x y0^2 (1 - x y0) the exact result is y0 (1 - e)^(-1/2) (y0 / (1 - e)), and the binomial
// (geometric) series is taken to e^2.  (One step of Householder's method of order two; A. S.
// Householder, The Numerical Treatment of a Single Nonlinear Equation, 1970.)
// On GB300 the FP64 pipe bounds the pair terms: 5 and 3 FP64 operations, and the seeds on the
// FP32 and special-function units; the conversions are integer operations.
#pragma once

#include <cuda_runtime.h>

namespace cutc {

// a double as a float, truncated, with integer operations (0 below the float range)
__device__ __forceinline__ float trunc_float(double x)
{
    const int hi = __double2hiint(x);
    const int v = (hi & 0x7fffffff) - 0x38000000;
    const unsigned m = ((unsigned)max(v, 0) << 3) | ((unsigned)__double2loint(x) >> 29);
    const unsigned f = v < 0x00100000 ? 0u : v >= 0x0ff00000 ? 0x7f7fffffu : m;
    return __uint_as_float(f | ((unsigned)hi & 0x80000000u));
}

// a positive normal float as a double, with integer operations
__device__ __forceinline__ double exact_double(float x)
{
    const unsigned b = __float_as_uint(x);
    return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

// 1/sqrt(x) for 2^-120 < x < 2^120.  The seed is within 2^-21.5 (truncation 2^-24 of the
// result, rsqrtf 2 ulp), |e| < 2^-20.5, so the series stops 5/16 e^3 < 2^-63 short; with the
// roundings of x y0 and of the sum the result is within 2^-52.
__device__ __forceinline__ double rsqrt_series(double x)
{
    const double y0 = exact_double(rsqrtf(trunc_float(x)));
    const double e = fma(-(x * y0), y0, 1.0);
    return fma(e * y0, fma(e, 0.375, 0.5), y0);
}

// 1/x for 2^-120 < x < 2^120.  The seed is within 2^-22.5 (truncation 2^-23, division 2^-24),
// so the series stops e^3 < 2^-66 short; e rounds at 2^-75, and the result is within 2^-52.9.
__device__ __forceinline__ double recip_series(double x)
{
    const double z0 = exact_double(__frcp_rn(trunc_float(x)));
    const double e = fma(-x, z0, 1.0);
    return fma(z0, fma(e, e, e), z0);
}

}  // namespace cutc
