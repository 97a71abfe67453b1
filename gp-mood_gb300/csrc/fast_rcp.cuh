// fast_rcp.cuh -- reciprocal and square root for the fast floating-point mode.
//
// Both correct the hardware's approximation once, with the residual's series
// to third order instead of two Newton steps: on this part an FP64 instruction
// costs an SM 16-19 cycles and a lone warp 64, so their number is what counts.
//
// 1/d from y ~ 1/d (PTX rcp.approx.ftz.f64): with e = 1 - d*y,
// 1/d = y/(1 - e) = y + y*(e + e^2) + O(e^3), the cubic ("hyperpower")
// iteration of M. Altman, Pacific J. Math. 10(4):1107-1113, 1960.  Measured
// |e| <= 2^-19.9, so the remainder is 2^-59.8: within an ulp or so of 1/d for
// normal d, not correctly rounded.  Three FP64 instructions; the two Newton
// steps it replaces took four, an IEEE division takes about seven and a half.
// A zero or subnormal d gives NaN.
//
// sqrt(x) from y ~ 1/sqrt(x) (PTX rsqrt.approx.ftz.f64): with g = x*y and
// e = 1 - g*y, sqrt(x) = g*(1 - e)^(-1/2) = g + g*e*(1/2 + 3/8 e) + O(e^3)
// (the binomial series).  Measured |e| <= 2^-19, remainder 2^-58.7.  Five FP64
// instructions and no branch (seven before); within an ulp or so for positive
// normal x, not correctly rounded.  Zero, negative and infinite x give NaN;
// the solver takes it only of a pressure over a density that it has already
// tested, or will test, for positivity.
#pragma once

__device__ __forceinline__ double gpm_fast_rcp(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double gpm_fast_sqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double g = x * y;
    const double e = fma(-g, y, 1.0);
    return fma(g * e, fma(0.375, e, 0.5), g);
}
