// FP64 inverse roots of squared distances.
#pragma once

#include "common.cuh"

namespace nbody {

// Whether r^-3 stays well inside the exponent range (false for zero, subnormal, NaN).
__device__ inline bool plain_range(double r2) { return (uint32_t)(__double2hiint(r2) >> 20) - 400u < 1250u; }

// The hardware's approximate r^-1 (y) and e = 1 - r^2 y^2, including what the rounding of
// r^2 y left. The instruction takes the upper word of r^2 alone and returns an upper word:
// over every upper word in [1, 4), with the lower word 0 and all ones, |e| <= 2^-19.03.
__device__ inline double approx_inverse(double r2, double &e) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
    const double h = __dmul_rn(r2, y);
    e = fma(-fma(r2, y, -h), y, fma(-h, y, 1.0));
    return y;
}

// Within plain_range: the approximation corrected by the binomial series of
// (1 - e)^(-1/2) = 1 + 1/2 e + 3/8 e^2 + ..., or, in the cube, of (1 - e)^(-3/2) =
// 1 + 3/2 e + 15/8 e^2 + ...; the next terms, 5/16 e^3 and 35/16 e^3, are below 2^-58.7
// and 2^-55.9.
__device__ inline double inverse_root(double r2) {
    double e;
    const double y = approx_inverse(r2, e);
    return fma(y, __dmul_rn(e, fma(e, 0.375, 0.5)), y);
}
__device__ inline double inverse_cube(double r2, double gm) {
    double e;
    const double y = approx_inverse(r2, e);
    const double p = __dmul_rn(gm, __dmul_rn(__dmul_rn(y, y), y));
    return fma(p, __dmul_rn(e, fma(e, 1.875, 1.5)), p);
}

}  // namespace nbody
