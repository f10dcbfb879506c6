// FP64 quotients, square roots and reciprocals, rounded as IEEE division and
// square root round them, without branches, for operands whose exponents are
// known to be moderate.
//
// The compiler's IEEE division and square root are calls that begin with a
// range test and end in a branch to a slow path; a particle-step of the MVS
// map makes forty of them, and the branches keep independent ones from
// overlapping. The sequences here take the hardware's coarse reciprocal or
// reciprocal square root (PTX rcp/rsqrt.approx.ftz.f64: 20-bit operands, low
// result word zero) and refine it with fused multiply-adds as Markstein does
// ("Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. R&D 34, 1990; "IA-64 and Elementary Functions", 2000): a
// third-order step to half an ulp, then one correction by the exact residual.
// The value before the last rounding is within 2^-103 of the true one, so the
// result is the IEEE one unless the true value lies that close to the middle
// of two doubles (an exact quotient or root always comes out exact). What is
// known of those: 2^36 random operands gave no difference; the reciprocals of
// roots that lie so close are a finite list, worked through (root_range);
// quotients made to lie there come out right where the reciprocal is known to
// half an ulp, and one in a hundred of them did not where it was a product of
// reciprocals, which therefore takes one more step (quotient_of). A quotient so
// small that its residual falls below the normal range may be an ulp off.
// A denominator that several quotients share pays for its reciprocal once,
// and sqrt and 1/sqrt share one seed.
//
// Operands must lie inside mid_range() (about 1e-60 .. 1e60 in magnitude), so that
// no product or residual leaves the normal range: one integer subtraction and
// compare. Zero, subnormal, infinite and NaN operands fail it: callers then run
// the plain statements.
#pragma once
#include <cuda_runtime.h>

namespace mb200 {

__device__ __forceinline__ double rcp_seed(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// True for positive x of binary exponent -200 .. 199 (sign, zero, infinity
// and NaN all fall outside: the high word is compared as an unsigned number).
__device__ __forceinline__ bool mid_range(double x) {
    return (unsigned)__double2hiint(x) - ((1023u - 200u) << 20) < (400u << 20);
}

// 1/b to half an ulp (and 2^-60): enough for quotient(), not yet rounded.
__device__ __forceinline__ double recip_near(double b) {
    const double y = rcp_seed(b);
    const double e = fma(-b, y, 1.0);
    return fma(fma(e, e, e), y, y);
}
// One residual correction of y ~ 1/b (within a few ulp): 1/b rounded.
__device__ __forceinline__ double recip_fix(double b, double y) { return fma(fma(-b, y, 1.0), y, y); }

// a/b rounded, from y = 1/b to half an ulp (and 2^-60): with y rounded this is
// Markstein's theorem, and the other y that recip_near and sqrt_near leave give
// no difference on quotients made to lie next to a middle.
__device__ __forceinline__ double quotient(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}
// a/b rounded, from y ~ 1/b (within a few ulp: a product of reciprocals). Without
// the step on y one in a hundred quotients made to lie next to a middle is an
// ulp off.
__device__ __forceinline__ double quotient_of(double a, double b, double y) { return quotient(a, b, recip_fix(b, y)); }
// a/b rounded, from a quotient q of it within an ulp and y as quotient()'s.
__device__ __forceinline__ double quotient_fix(double a, double b, double y, double q) {
    return fma(fma(-b, q, a), y, q);
}

__device__ __forceinline__ double half_of(double y) {  // y/2 of a normal y, on the integer pipe
    return __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
}

// s = sqrt(x) rounded; y = 1/sqrt(x) to half an ulp (and 2^-60).
__device__ __forceinline__ void sqrt_near(double x, double& s, double& y) {
    const double y0 = rsqrt_seed(x);
    const double e = fma(-x, y0 * y0, 1.0);  // y0 has 21 bits: its square is exact
    y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
    const double g = x * y;
    s = fma(fma(-g, g, x), half_of(y), g);
}
// s = sqrt(x) rounded and r = 1/s rounded: the two roundings of 1.0 / sqrt(x),
// for x inside root_range().
__device__ __forceinline__ void sqrt_recip(double x, double& s, double& r) {
    double y;
    sqrt_near(x, s, y);
    r = recip_fix(s, y);
}

// mid_range less the operands whose significand ends in 32 ones. One in 2^53
// of them, 4^k (1 - 2^-53), has a root whose reciprocal recip_fix gets wrong: the
// significand of the root is all ones, and the residual correction ends in the
// middle of two doubles. The other reciprocals that lie as close to a middle as
// the correction's error (the 53-bit factors of 2^106 - 16 .. 2^106 + 16) were
// worked through one by one and come out right.
__device__ __forceinline__ bool root_range(double x) { return mid_range(x) && __double2loint(x) != -1; }

// The same for any operands: what is out of range takes the plain statements,
// by a call (their code then stays out of the way of the code around).
static __device__ __noinline__ double sqrt_plain(double x) { return sqrt(x); }
static __device__ __noinline__ double div_plain(double a, double b) { return a / b; }
__device__ __forceinline__ void sqrt_recip_any(double x, double& s, double& r) {
    sqrt_recip(x, s, r);
    if (!root_range(x)) {
        s = sqrt_plain(x);
        r = div_plain(1.0, s);
    }
}
__device__ __forceinline__ bool mid_magnitude(double x) {   // mid_range of |x|
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) - ((1023u - 200u) << 20) < (400u << 20);
}

}  // namespace mb200
