// lg_house.cuh -- one Householder reflector (LAPACK dlarfg conventions) from
// plain sums of squares, shared by the panel, TSQR and batched kernels.
//
// The kernels form sum(x^2) without dlarfg's scaling (a maximum and a division
// per element on the narrow FP64 pipe) and ask house_in_range; a column that
// answers no is scaled by 2^-house_shift (from its largest exponent, integer
// work) and taken again, its beta scaled back.
#pragma once

#include <math.h>

#include "lg_common.cuh"

namespace lg {

// H = I - tau v v^T = I - tau sc^2 u u^T with v = sc u, u the column with its
// pivot entry replaced by alpha - beta.
struct Reflector {
    double beta, tau, sc, u;
};

// The biased exponent of x (an FP64 compare would hold the pipe for 64 clocks).
__device__ __forceinline__ int bexp_of(double x) { return (__double2hiint(x) >> 20) & 0x7FF; }

// Whether alpha^2 + ss and ss are safely inside the FP64 range (2^+-930).
__device__ __forceinline__ bool house_in_range(double alpha, double ss)
{
    return bexp_of(ss) >= 1023 - 930 && bexp_of(fma(alpha, alpha, ss)) <= 1023 + 930;
}

// x / 2 for a normal x whose half is normal: an exponent move.
__device__ __forceinline__ double half_of(double x)
{
    return __hiloint2double(__double2hiint(x) - (1 << 20), __double2loint(x));
}

// The reflector by square root and divisions, for sums outside the range above
// (non-finite ones among them).  Out of line: inline, the compiler issues part
// of it for every column.
static __device__ __noinline__ Reflector house_reflector_wide(double alpha, double s)
{
    const double beta = -copysign(sqrt(s), alpha);
    return Reflector{beta, (beta - alpha) / beta, 1.0 / (alpha - beta), alpha - beta};
}

// dlarfg from the pivot alpha and the sum of squares below it; `below` says
// whether anything below the pivot is nonzero.  |beta| = sqrt(alpha^2 + ss)
// corrected to rounding level, tau = 1 + |alpha| / |beta|, sc = 1 / (alpha -
// beta): 16 dependent FP64 operations against ~45 of sqrt and two divisions.
// (What is not FP64 counts too: with the seeds formed in single precision and
// moved by integer instructions the reflector took 2,700 clocks of a column's
// chain, where the 16 operations take 1,030.)
__device__ __forceinline__ Reflector house_reflector(double alpha, double ss, bool below)
{
    if (!below) return Reflector{alpha, 0.0, 0.0, 0.0};
    const double s = fma(alpha, alpha, ss), a = fabs(alpha);
    const int ex = bexp_of(s);
    if (ex >= 1023 - 960 && ex <= 1023 + 960) {
        const double y = rsqrt_normal(s);
        double b = s * y;
        b = fma(half_of(y), fma(-b, b, s), b);
        const double t = b + a;
        double tau = t * y;
        tau = fma(fma(-tau, b, t), y, tau);
        return Reflector{-copysign(b, alpha), tau, copysign(rcp_nr(t), alpha), copysign(t, alpha)};
    }
    return house_reflector_wide(alpha, s);
}

// Biased exponent + 64 of x's leading bit (0 for x = 0), so that subnormals
// order below the normal numbers.
__device__ __forceinline__ int house_exponent(double x)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(x) << 1;
    const int ex = (int)(u >> 53);
    return u ? (ex ? ex + 64 : 75 - __clzll((long long)u)) : 0;
}

// The power of two of a column's largest house_exponent (0: nothing to scale,
// a zero or non-finite column).
__device__ __forceinline__ int house_shift(int e) { return (e == 0 || e >= 0x7FF + 64) ? 0 : e - 64 - 1023; }

// Sum over groups of LG lanes.
template <int LG>
__device__ __forceinline__ double group_sum(double v)
{
#pragma unroll
    for (int o = LG / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace lg
