// rsqrt64.cuh -- x^(-1/2) and x^(-3/2) in FP64 for the pair sums.
//
// The all-pairs FP64 kernels are bound by the FP64 pipe, and most of a pair's FP64 instructions would be the
// library's square root and division (about 60 of 75). Here one hardware approximation
// (rsqrt.approx.ftz.f64, PTX ISA) gives y with x y^2 = 1 - e, |e| < 2^-18, and the binomial series
// (1 - e)^(-s) = 1 + s e + s (s + 1) / 2 e^2 + ..., s = 1/2 or 3/2, cut after the e^2 term, does the rest: 5 and 6
// FP64 instructions, truncation below 2.2 |e|^3 < 2^-52. y carries at most 21 significant bits, so y^2 is exact.
#pragma once

#include <cuda_runtime.h>

namespace gsph {

// 2^-600 <= x < 2^600, by the exponent bits: no intermediate of the series over- or underflows. False for
// zero, negative, infinite and NaN x, which take the library's functions.
__device__ __forceinline__ bool series_range64(double x) {
    return static_cast<unsigned>(__double2hiint(x)) - 0x1a700000u < 0x4b000000u;
}
__device__ __forceinline__ double rsqrt_seed64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double inv_sqrt64(double x) {  // x^(-1/2), series_range64(x)
    const double y = rsqrt_seed64(x);
    const double e = fma(-x, y * y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ double inv_cube64(double x) {  // x^(-3/2), series_range64(x)
    const double y = rsqrt_seed64(x);
    const double t = y * y;
    const double e = fma(-x, t, 1.0);
    const double y3 = t * y;
    return fma(y3 * e, fma(1.875, e, 1.5), y3);
}

}  // namespace gsph
