// rsqrt64.cuh — inverse distances in double precision for the FP64 sums.
//
// The hardware's approximation y of 1/sqrt(x) has |h| < 2^-19 in
// h = 1 - x y^2 (measured: 2^-19.14 over 2^-300..2^300; y has 20 mantissa
// bits, so y^2 is exact and h is rounded once).  1/sqrt(x) = y (1 - h)^(-1/2)
// and its cube follow from the binomial series, whose first term left out is
// 5/16 h^3 < 2^-58 and 35/16 h^3 < 2^-55: below the rounding of a double sum's
// terms, in 6 and 7 operations.
//
// Both hold for finite m and normal, finite x.  Anything else (a distance of 0
// or infinity, a softening whose square is subnormal, a mass that is not
// finite) comes out infinite or NaN, never as a wrong finite number, so a sum
// that is finite is right and one that is not is taken again with rsqrt().
#pragma once

__device__ __forceinline__ double rsqrt64_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// m / x^(3/2)
__device__ __forceinline__ double mass_over_r3(double m, double x) {
    const double y = rsqrt64_seed(x), y2 = y * y;
    const double h = fma(-x, y2, 1.0);
    const double f = (m * y) * y2;
    return fma(f, h * fma(1.875, h, 1.5), f);
}

// m / sqrt(x)
__device__ __forceinline__ double mass_over_r(double m, double x) {
    const double y = rsqrt64_seed(x);
    const double h = fma(-x, y * y, 1.0);
    const double f = m * y;
    return fma(f, h * fma(0.375, h, 0.5), f);
}
