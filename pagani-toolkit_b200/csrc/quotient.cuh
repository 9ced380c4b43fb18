// quotient.cuh -- FP64 quotients without a branch, so that several run side by
// side: Newton steps on the quotient with exact remainders (P. Markstein, IBM
// J. Res. Dev. 34(1), 1990).  Each is the correctly rounded quotient on the
// range that it names (tests/test_quotients_gpu.py compares them with the
// division operator).
#pragma once
#include <cuda_runtime.h>

// a / b for normal b and a normal or zero a whose quotient is normal or zero:
// the reciprocal by Newton's iteration from the hardware's approximation, then
// two quotient corrections.  Newton's iteration ends in the correctly rounded
// reciprocal but for one mantissa, all ones: 1 / b lies just above the middle
// of a power of two and its successor, and the iteration may stop at the
// former.  The successor is put in there (otherwise 1 / (1 - 2^-53) came out as 1,
// and the Fisher transform of an r of 6e-17 as 0).
__device__ __forceinline__ double div_normal(double a, double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    constexpr unsigned long long ONES = 0xfffffffffffffULL;
    const unsigned long long last = ((unsigned long long)__double_as_longlong(b) & ONES) == ONES;
    y = __longlong_as_double((long long)((unsigned long long)__double_as_longlong(y) | last));
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// x / d for r = 1 / d rounded to nearest, x and x / d below 2^400 in magnitude
// and a d that div_by_divisor admits (an entry by its vector's norm, a sum by a
// count).  x is scaled so that no remainder underflows: without that, quotients
// of an x below 2^-968 could be an ulp off.  A quotient below the normal numbers is rounded twice (its
// last bit may differ from the operator's); a zero has either sign.
__device__ __forceinline__ double div_by(double x, double d, double r)
{
    const double xs = __dmul_rn(x, 0x1p+600);
    double q = __dmul_rn(xs, r);
    q = __fma_rn(__fma_rn(-d, q, xs), r, q);
    return __dmul_rn(__fma_rn(__fma_rn(-d, q, xs), r, q), 0x1p-600);
}
__device__ __forceinline__ bool div_by_divisor(double d) { return d > 0x1p-200 && d < 0x1p+200; }
