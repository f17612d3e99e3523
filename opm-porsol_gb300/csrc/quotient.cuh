// quotient.cuh -- FP64 quotients in few operations, for kernels bound by the FP64 pipe (two operations a clock
// and SM on GB300, where a division is a sequence of a dozen).
//
// Both start from the hardware's estimate of the reciprocal (rcp.approx.ftz.f64, about 20 bits) and refine it by
// Newton-Raphson steps (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor",
// IBM J. Res. Dev. 34, 1990).  The estimate flushes subnormals: denominators below 2^-1022 or of 2^1022 and above,
// zeros, infinities and NaN take the division instead, chosen on the integer pipe.
#pragma once

namespace porsol {

// exponent field in [1, 0x7fc]: 2^-1022 <= |x| < 2^1022
__device__ __forceinline__ bool estimable(double x)
{
    return unsigned((__double2hiint(x) >> 20 & 0x7ff) - 1) < 0x7fcu;
}

__device__ __forceinline__ double reciprocal_estimate(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    return r;
}

// num / den, within an ulp of the rounded quotient (num 0 or at least 2^-960 in size; below that the
// remainder underflows): one Newton step (40 bits) and the quotient corrected once by its remainder
__device__ __forceinline__ double quotient(double num, double den)
{
    if (!estimable(den)) return num / den;
    double r = reciprocal_estimate(den);
    r = fma(r, fma(-den, r, 1.0), r);
    const double q = num * r;
    return fma(fma(-den, q, num), r, q);
}

// 1 / x, within an ulp of the rounded reciprocal: two Newton steps
__device__ __forceinline__ double reciprocal(double x)
{
    if (!estimable(x)) return 1.0 / x;
    double r = reciprocal_estimate(x);
    r = fma(r, fma(-x, r, 1.0), r);
    return fma(r, fma(-x, r, 1.0), r);
}

}  // namespace porsol
