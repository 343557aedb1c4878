/*
 * quotient.cuh — IEEE quotients of the FP64 cable solve without a division's branches (a dependent
 * division measured 127 cycles on a B200, an FP64 fma 8.6, rcp.approx.ftz.f64 17.7), after
 * P. W. Markstein, "Computation of elementary functions on the IBM RISC System/6000
 * processor", IBM J. Res. Dev. 34(1), 1990, and J.-M. Muller et al., Handbook of
 * Floating-Point Arithmetic, chapter on FMA-based division:
 *   - two Newton steps on a seed good to 2^-19 leave y2 within one unit in the last place of
 *     1/D, and a third, y3 = y2 + y2 (1 - D y2) with the residual exact in one FMA, rounds to
 *     the nearest double of 1/D, unless D's significand is all ones;
 *   - q1 = q0 + (n - D q0) y is within one unit in the last place of n/D, its residual
 *     r1 = n - D q1 is exact, and q1 + r1 y3 rounds to the IEEE quotient.
 *
 * The residuals are exact while nothing overflows or loses bits to underflow.  good_divisor,
 * good_axial and good_quotient say where that is known to hold, from the operands that the solve
 * still has when it is done: its pivots D, the axial terms a, and the solution x = n/D.
 *   - D in [2^-480, 2^480), significand not all ones;
 *   - a / D: a zero or in [2^-480, 2^480), so the residual's last bit is above 2^-586;
 *   - n / D: x normal, and the sum of x's and D's exponents at least -959: n is then at least
 *     about 2^-960 and the residual's last bit at least 2^-1064, where the smallest double is
 *     2^-1074.  A zero x came from a zero n, or from one so small that n/D rounds to zero
 *     as well: n y only rounds to zero where n/D does, unless D's significand is all ones.
 * -0 as a numerator gives +0; the solve has none: its sums start at +0.
 */
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

namespace mind {

__host__ __device__ __forceinline__ uint64_t magnitude_bits(double x) {
    uint64_t u;
#ifdef __CUDA_ARCH__
    u = (uint64_t)__double_as_longlong(x);
#else
    std::memcpy(&u, &x, sizeof u);
#endif
    return u & 0x7FFFFFFFFFFFFFFFull;
}
/* Biased exponent and the top 20 fraction bits of |x|. */
__host__ __device__ __forceinline__ uint32_t magnitude_high(double x) { return (uint32_t)(magnitude_bits(x) >> 32); }

/* 2^low <= |x| < 2^high (low > -1023, high <= 1024). */
__host__ __device__ __forceinline__ bool in_binades(double x, int low, int high) {
    return magnitude_high(x) - ((uint32_t)(1023 + low) << 20) < (uint32_t)(high - low) << 20;
}

__host__ __device__ __forceinline__ bool good_divisor(double D) {
    return in_binades(D, -480, 480) && ((magnitude_bits(D) + 1) & 0xFFFFFFFFFFFFFull) != 0;
}
__host__ __device__ __forceinline__ bool good_axial(double a) { return a == 0.0 || in_binades(a, -480, 480); }
/* x = n / D, D a good divisor. */
__host__ __device__ __forceinline__ bool good_quotient(double x, double D) {
    return x == 0.0 || (in_binades(x, -1000, 400) && magnitude_high(x) + magnitude_high(D) >= (uint32_t)(2046 - 958) << 20);
}
/* Both, from the high words and for all but odd values: |x| at least 2^-400, D's significand not
 * starting with twenty ones. */
__host__ __device__ __forceinline__ bool surely_good(double D, double x) {
    return in_binades(D, -480, 480) && ((magnitude_high(D) + 1) & 0xFFFFFu) != 0 && (x == 0.0 || in_binades(x, -400, 400));
}

__host__ __device__ __forceinline__ double reciprocal_seed(double D) {
    double y;
#ifdef __CUDA_ARCH__
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(D));
#else   // for tests on the CPU: the instruction's documented operand and result, 20 fraction bits each
    uint64_t u;
    std::memcpy(&u, &D, sizeof u);
    u &= ~0xFFFFFFFFull;
    std::memcpy(&y, &u, sizeof y);
    y = 1.0 / y;
    std::memcpy(&u, &y, sizeof u);
    u &= ~0xFFFFFFFFull;
    std::memcpy(&y, &u, sizeof y);
#endif
    return y;
}
__host__ __device__ __forceinline__ double reciprocal(double D) {
    double y = reciprocal_seed(D);
    y = fma(y, fma(-D, y, 1.0), y);
    y = fma(y, fma(-D, y, 1.0), y);
    return fma(y, fma(-D, y, 1.0), y);
}
/* n / D from D's reciprocal. */
__host__ __device__ __forceinline__ double quotient(double n, double D, double y) {
    const double q0 = n * y;
    const double q1 = fma(fma(-D, q0, n), y, q0);
    return fma(fma(-D, q1, n), y, q1);
}
/* a / D with D just known: the quotient starts from the reciprocal's first iterate. */
__host__ __device__ __forceinline__ double pivot_quotient(double a, double D) {
    const double y0 = reciprocal_seed(D);
    const double y1 = fma(y0, fma(-D, y0, 1.0), y0);
    const double q0 = a * y1;
    const double y2 = fma(y1, fma(-D, y1, 1.0), y1);
    const double q1 = fma(fma(-D, q0, a), y2, q0);
    const double y3 = fma(y2, fma(-D, y2, 1.0), y2);
    return fma(fma(-D, q1, a), y3, q1);
}

}  // namespace mind
