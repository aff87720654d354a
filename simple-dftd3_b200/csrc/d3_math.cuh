// Reciprocals, reciprocal square roots and even powers of the pair terms.
//
// FP64: the hardware approximation y (relative error e0 below 2^-20) and one
// third-order Householder step: with the residual e = 1 - x y (1 - x y^2) the result
// is y (1 - e)^-1 (y (1 - e)^-1/2), its binomial series cut after e^2, error of order
// e0^3 = 2^-60, below the rounding.  4 and 6 instructions without branches, in
// place of the library's division and square root with their special cases; within
// one and two units in the last place for normal arguments whose result is normal.
// An infinite argument gives NaN: the callers' arguments are squared distances and
// sums of positive terms far from the ends of the range, and the powers of the
// damping functions, which are not, are bounded first (damping_power).  Measured (B200, FP64): the CN sweep of a
// periodic 2000-atom cell 161 -> 108 us (two divisions and a square root less per
// term), its rational two-body sweep 232 -> 210 us, the optimized power sweep of a
// 141-atom slab 247 -> 114 us (no pow).
#pragma once

#include <cuda_runtime.h>

namespace d3 {

__device__ __forceinline__ double rcp_fast(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = ::fma(-x, y, 1.0);
    return ::fma(y, ::fma(e, e, e), y);
}

// 1/x in FP32: the hardware approximation (1 ulp).
__device__ __forceinline__ float rcp_fast(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ double rsqrt_fast(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = ::fma(-x * y, y, 1.0);
    return ::fma(y * e, ::fma(e, 0.375, 0.5), y);
}

// 1/x in the precision of the form: FP64 as above, FP32 correctly rounded.
template <class R>
__device__ __forceinline__ R inv(R x) { if constexpr (sizeof(R) == 8) return rcp_fast(x); else return 1.0f / x; }

// Half of an even exponent 2 h with 0 <= h <= 32, else -1: (q / r)^alp is then
// (q^2 / r^2)^h by squarings (7 multiplications at the usual exponents of 14 and
// 16), without square root, log and exp.  The factors carry as many roundings as
// the power magnifies the one of q / r.
__device__ __forceinline__ int half_even(double alp)
{
    const int h = (int)(0.5 * alp);
    return h >= 0 && h <= 32 && 2.0 * h == alp ? h : -1;
}

// x^h for 0 <= h <= 32 (the same h in all lanes)
template <class R>
__device__ __forceinline__ R ipow(R x, int h)
{
    R y = R(1);
    while (h) {
        if (h & 1) y *= x;
        h >>= 1;
        if (h) x *= x;
    }
    return y;
}

// A damping power t = (R0/r)^alp (r^-bet), bounded so that 1 + 6 t, 6 alp t (R0^(bet + 8) t) stay finite for any
// exponent and distance (the rejected terms of a sweep take r = 1, where a large alp
// overflows first): the damping 1 / (1 + 6 t) has vanished long before.
template <class R>
__device__ __forceinline__ R damping_power(R t) { if constexpr (sizeof(R) == 8) return fmin(t, 1e150); else return fminf(t, 1e30f); }

}  // namespace d3
