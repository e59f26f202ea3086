// FP64 inverse square root without branches, for the accurate walks: rsqrt()
// carries one for its special operands in every call, which ends the basic
// block, and these walks are bound by the latency of their dependent FP64
// operations -- without it the compiler interleaves several interactions.
#pragma once

namespace nb {

// x^(-1/2) by Householder's third-order iteration from PTX's approximate seed
// (20 bits; 9e-7 measured), for normal x.  Largest relative error 1.1e-16
// against 80-bit roots (1.0 / sqrt(x): 1.7e-16), held to 1.15e-16 over
// 2^-958 .. 2^960 by the tests.
__device__ __forceinline__ double rsqrt_fast(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y * y, 1.0);                     // x y^2 = 1 - e; y y is exact, y being short
    return fma(y * e, fma(e, 0.375, 0.5), y);                 // y (1 + e/2 + 3 e^2 / 8)
}

// x with its exponent kept within 2^-960 .. 2^960: rsqrt_fast's operand where
// it may be zero, infinite or nearly so (a force from there is zero either way).
// Beyond a limit the low half of the mantissa stays: at most 2^-20 off the limit.
__device__ __forceinline__ double away_from_ends(double x) {
    const int hi = min(max(__double2hiint(x), 0x03f00000), 0x7bf00000);
    return __hiloint2double(hi, __double2loint(x));
}

}  // namespace nb
