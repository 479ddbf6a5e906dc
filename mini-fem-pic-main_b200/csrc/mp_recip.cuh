// The reciprocal on the sparse factorization's chain of pivots, where a division's
// latency would be.
#pragma once

namespace mp {

// Whether reciprocal(d) holds its bound: 2^-960 <= |d| < 2^961 (by the exponent alone).
__device__ __forceinline__ bool invertible(double d) {
    return (unsigned)((__double2hiint(d) >> 20 & 0x7ff) - (1023 - 960)) <= 2 * 960;
}

// 1/d by the hardware approximation x (e = 1 - d x, |e| below 2^-20) and one step of the
// third-order Householder iteration, x (1 + e + e^2): what is left out is e^3, so the
// result is within 2^-53 (1 + 2^-6) of 1/d, relative, for an invertible d.
__device__ __forceinline__ double reciprocal(double d) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
    const double e = fma(-d, x, 1.0);
    return fma(x, fma(e, e, e), x);
}

}  // namespace mp
