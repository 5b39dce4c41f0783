// ieee64.h -- correctly rounded FP64 quotients and square roots without
// branches, for the FP64 stage kernels.
//
// The `/` and sqrt() of the device are correctly rounded too, but each one
// carries a test and a call for its special operands (zeros among them, the
// common operand of still water and dry land), which splits the code into
// basic blocks: no two of the ~70 divisions and roots of a cell-stage overlap,
// and the chain of dependent FP64 instructions bounds the kernel.  Here a
// caller checks the exponents of a whole group of operands once (mid /
// mid_or_zero), evaluates the group in one straight line, and falls back to
// the ordinary operators when the check fails.  Quotients by the same divisor
// share its reciprocal.
//
//  * reciprocal: Newton-Raphson from a seed, y <- y + y (1 - d y) with the
//    residual in one fused multiply-add.  From a seed good to 2^-19 two steps
//    leave y within an ulp of 1/d; the third makes it the correctly rounded
//    reciprocal, except for a divisor whose significand is all ones
//    (P. Markstein, "Computation of elementary functions on the IBM RISC
//    System/6000 processor", IBM J. Res. Dev. 34, 1990, theorems 7-8).
//    recip_ok() sends those divisors to the fallback.
//  * quotient: q0 = a y, two corrections q <- q + y (a - d q).  The first
//    leaves q faithful; the second, with a correctly rounded y and the exact
//    residual of a faithful q, gives the correctly rounded quotient (same
//    source, theorem 8's corollary).  Operands between 2^-800 and 2^800 whose
//    quotient lies between 2^-1000 and 2^1000 keep every intermediate result
//    and residual in the normal range; mid() tests the operands, and the bound
//    on the quotient follows at each call site from what its divisor can be.
//  * square root: the coupled iteration g -> sqrt(x), h -> 1/(2 sqrt(x)),
//    r = 1/2 - g h, g <- g + g r, h <- h + h r (R. Goldschmidt, 1964), then
//    g <- g + h (x - g^2).  After two steps g is within 0.51 ulp and h within
//    2^-53; the last step then lands within 2^-53.6 ulp of the root.  A root
//    of a 53-bit x lies at least 2^-53.2 ulp from any rounding boundary except
//    for significands next to a power of four (x = k (k + 1) in units of the
//    last place), so the result is correctly rounded.
// tests/ieee64_check.cpp checks both against the host's IEEE operations on
// random operands, on the operands whose roots lie closest to a rounding
// boundary, and over the seeds' error range; tests/ieee64_device_check.cu the
// device's own seeds (their error and the results) against its `/` and sqrt.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define TSU_HD __host__ __device__ __forceinline__
#else
#define TSU_HD inline
#endif

namespace tsu {

TSU_HD double fma64(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
TSU_HD uint32_t hi32(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return (uint32_t)(u >> 32);
#endif
}
TSU_HD uint32_t lo32(double x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    std::memcpy(&u, &x, 8);
    return (uint32_t)u;
#endif
}

// 2^-800 <= |x| < 2^800 (false for zeros, infinities and NaN)
TSU_HD bool mid(double x) { return (hi32(x) & 0x7fffffffu) - 0x0df00000u < 0x64000000u; }
// the same, or a zero
TSU_HD bool mid_or_zero(double x) {
    const uint32_t t = hi32(x) & 0x7fffffffu;
    return (t - 0x0df00000u < 0x64000000u) | ((t | lo32(x)) == 0u);
}
// 2^-800 <= |x| < 2^80, or a zero
TSU_HD bool small_or_zero(double x) {
    const uint32_t t = hi32(x) & 0x7fffffffu;
    return (t - 0x0df00000u < 0x44f00000u - 0x0df00000u) | ((t | lo32(x)) == 0u);
}
// The significand of a divisor is not all ones, judged by its low word (a few
// other divisors take the fallback too).
TSU_HD bool recip_ok(double d) { return lo32(d) != 0xffffffffu; }

// RN(1/d) from a seed y with |y d - 1| <= 2^-19; mid(d), recip_ok(d)
TSU_HD double recip_from(double d, double y) {
    double e = fma64(-d, y, 1.0);
    y = fma64(y, e, y);
    e = fma64(-d, y, 1.0);
    y = fma64(y, e, y);
    e = fma64(-d, y, 1.0);
    return fma64(y, e, y);
}
// RN(a/d) from y = RN(1/d) and a first quotient q0 with |q0 d / a - 1| <= 2^-30
// (the first correction leaves any such q0 faithful); mid_or_zero(a) (a zero
// numerator gives a zero, its sign not kept)
TSU_HD double quot_from(double a, double d, double y, double q0) {
    double r = fma64(-q0, d, a);
    const double q = fma64(r, y, q0);
    r = fma64(-q, d, a);
    return fma64(r, y, q);
}
TSU_HD double quot(double a, double d, double y) { return quot_from(a, d, y, a * y); }
// RN(sqrt(x)) from a seed y with |y sqrt(x) - 1| <= 2^-19; mid(x), x > 0
TSU_HD double sqrt_from(double x, double y) {
    double g = x * y, h = 0.5 * y;
    double r = fma64(-g, h, 0.5);
    g = fma64(g, r, g);
    h = fma64(h, r, h);
    r = fma64(-g, h, 0.5);
    g = fma64(g, r, g);
    h = fma64(h, r, h);
    const double d = fma64(-g, g, x);
    return fma64(d, h, g);
}

#ifdef __CUDACC__
// The seeds: PTX's approximate reciprocal and reciprocal square root.
__device__ __forceinline__ double recip(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    return recip_from(d, y);
}
// x >= 0, mid_or_zero(x).  A zero gets a finite seed, whose iterates stay 0.
__device__ __forceinline__ double root(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    y = __hiloint2double(__double2hiint(x) ? __double2hiint(y) : 0x3ff00000, __double2loint(y));
    return sqrt_from(x, y);
}
#endif

}  // namespace tsu
