// ieee64.cuh -- correctly rounded FP64 quotients and square roots as straight-line code, for the flux
// kernels of the plain path.
//
// The compiler's / and sqrt branch to an out-of-line routine for operands outside their fast range, and
// a zero numerator or argument is outside it: in a flow with a quiescent ambient (zero velocities, equal
// pressures, equal densities in both logarithmic means) most divisions of a stage took that branch.
// Here a quotient is Markstein's (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34 (1990); M. Cornea, J. Harrison, P. T. P. Tang, "Scientific
// Computing on Itanium-based Systems" (2002)): y ~ 1/b by two Newton steps, q = RN(a y), r = a - b q
// (exact with one FMA), RN(q + r y).  Next to a rounding tie of a/b the first quotient q is off by exactly
// half an ulp, so the corrected sum errs by less than the distance of a/b from the tie, given y to half
// an ulp.  Newton's steps miss that half ulp only where 1/b lies within 2^-80 of a tie, foremost for a
// significand of all ones (1 - 2^-53 and its multiples by powers of two, a density a hair below 1), whose
// reciprocal is set directly.  Quotients by the same b share y: three operations each.  The square root
// is the same idea on y ~ 1/sqrt(a): g = RN(a y), RN(g + (a - g^2) y/2).
//
// Domain: operands, results and their products with a few ulp's worth of residual in the normal range
// (|a| zero or above about 1e-290, |b| from 2^-1000 to 2^1000); the square root's argument likewise.  A zero
// quotient comes back as +0.  Outside, a last bit is lost, a zero or infinite denominator and an infinite numerator
// give NaN: callers see to it that no operand is (regular64 in euler_fp64.cuh), or take Plain64.  Same bits as /
// and sqrt inside (tests/test_gpu_fp64_domain.py: quotients next to a rounding tie, significands of all ones,
// the neighbourhoods of powers of two, random operands over the whole domain).
// What they give: the stage kernel of stage_fp64.cu, Sedov 32^3, 727 us with / and sqrt (340 M warp
// instructions), 381 us with these and 24 warps per SM (242 M).
#pragma once

namespace nemo {

struct Rcp64 {
    double b, y;   // y = 1/b to the last bit (rounded to nearest except next to a tie)
};

__device__ __forceinline__ Rcp64 rcp64r(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));   // relative error below 2^-20
    y = fma(y, fma(-b, y, 1.0), y);
    y = fma(y, fma(-b, y, 1.0), y);
    // all ones: 1/b = (1 + 2^-53 + 2^-106 + ...) 2^k, just above the tie; Newton stops at 2^k
    if ((__double2loint(b) & (__double2hiint(b) | (int)0xfff00000)) == -1)
        y = __hiloint2double(__double2hiint(y), __double2loint(y) | 1);
    return {b, y};
}

__device__ __forceinline__ double quot64(double a, const Rcp64& r) {
    const double q = a * r.y;
    return fma(fma(-r.b, q, a), r.y, q);
}

__device__ __forceinline__ double div64(double a, double b) { return quot64(a, rcp64r(b)); }

__device__ __forceinline__ double sqrt64(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);                  // y (1 + e/2 + 3 e^2/8) ~ 1/sqrt(a)
    y = fma(fma(e, 0.375, 0.5), y * e, y);
    const double g = a * y;
    const double s = fma(fma(-g, g, a), 0.5 * y, g);
    return a == 0.0 ? a : s;
}

// The two arithmetics of a flux: the quotients above, for operands inside their domain, and the language's own
// for any operands.
struct Quick64 {
    static __device__ __forceinline__ Rcp64 rcp(double b) { return rcp64r(b); }
    static __device__ __forceinline__ double quot(double a, const Rcp64& r) { return quot64(a, r); }
    static __device__ __forceinline__ double div(double a, double b) { return div64(a, b); }
    static __device__ __forceinline__ double root(double a) { return sqrt64(a); }
};
struct Plain64 {
    static __device__ __forceinline__ Rcp64 rcp(double b) { return {b, 0.0}; }
    static __device__ __forceinline__ double quot(double a, const Rcp64& r) { return a / r.b; }
    static __device__ __forceinline__ double div(double a, double b) { return a / b; }
    static __device__ __forceinline__ double root(double a) { return sqrt(a); }
};

}  // namespace nemo
