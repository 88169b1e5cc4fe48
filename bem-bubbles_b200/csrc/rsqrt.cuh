// The FP64 reciprocal square root of the pair loops.
#pragma once

namespace bemb {

// 1/sqrt(r2) for r2 > 0 in FP64: the hardware's approximate reciprocal square root
// (rsqrt.approx.ftz.f64) refined by the binomial series of (1-d)^(-1/2) = 1 + d/2 + 3d^2/8 + ...
// with d = 1 - r2*y0^2; truncation error 5d^3/16, far below the double rounding unit for the
// estimate's relative error.  The estimate has the upper 32 bits of a double only, so y0^2 is exact.
__device__ __forceinline__ double rsqrt_fp64(double r2) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(r2));
    const double d = fma(-r2, __dmul_rn(y0, y0), 1.0);
    const double p = fma(0.375, d, 0.5);
    return fma(y0, __dmul_rn(d, p), y0);
}

}  // namespace bemb
