// Straight-line FP64 division and square root for the solvers of the FP64 path.
//
// The FP64 kernels are bound by the latency of dependent FP64 instructions at 4 warps per
// scheduler.  An IEEE `a / b` or sqrt(x) of double compiles to a sequence with a branch to a
// slow path, and the branches keep independent quotients from overlapping: each one's whole
// latency is exposed.  Here each operation is a fixed sequence of multiply-adds with no branch,
// several quotients share the reciprocal of a common divisor, and the operands' exponents are
// collected in two integers that a solve tests once at its end; a solve with an operand outside
// the safe range is done again with the IEEE operators (the callers' *_ieee functions).
//
// Methods (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990; J.-M. Muller et al., "Handbook of Floating-Point
// Arithmetic", chapter 4).  Reciprocal: an approximation y of 1/b within an ulp, rounded up, then
// RN(y + y (1 - b y)), which is RN(1/b) (rounded up first, because from below the divisor whose
// significand is all ones ends in a tie).  Quotient: q = RN(a y), the exact remainder r = b q - a,
// RN(q - r y): with y = RN(1/b) and q within an ulp this is RN(a/b).  Square root: g within an ulp,
// rounded down, z = 1/sqrt(x), the exact d = x - g^2, RN(g + d z / 2).
//
// The last rounding sees the true value to 2^-52 ulp or so, and operands a few ulps from a power of
// two (a density of 1 - 2^-53, say) do lie that close to a tie: the directed roundings above put the
// error on the side away from it.  What is left are quotients whose first q is off by more than an
// ulp (a's significand below b's) and which also lie within 2^-53 ulp of a tie, about one in 1e17.
// Compared with the operators on 2e10 random operand pairs and on every pair of significands within
// 12 ulps of 1, 1.25, 1.5, 1.75 and their powers of two: no difference.
//
// Seeds: the PTX instructions rcp.approx.ftz.f64 and rsqrt.approx.ftz.f64 (measured relative error
// 1e-6); one step of third order takes them to the last bit.
//
// Signs of zero quotients are IEEE's for positive divisors (r is formed as b q - a, so that
// q - r y keeps a zero's sign); a negative divisor counts as out of range, and callers that
// divide by a negative quantity divide the negated numerator by its negative instead.
#pragma once
#include <cuda_runtime.h>

namespace dg {

// The operators themselves, behind the same interface: the reference form of every solve.
struct IeeeMath {
    static constexpr bool kZeroTest = true;  // a solve tests a divisor that may be zero itself
    struct Rec {};
    __device__ __forceinline__ Rec rec(double) { return Rec{}; }
    __device__ __forceinline__ double div(double a, double b, Rec) { return a / b; }
    __device__ __forceinline__ double inv(double b) { return 1.0 / b; }
    __device__ __forceinline__ double root(double x) { return sqrt(x); }
    // s = sqrt(x) and what div() needs to divide by s
    __device__ __forceinline__ double root(double x, Rec &) { return sqrt(x); }
    __device__ __forceinline__ double inv_root(double x) { return 1.0 / sqrt(x); }
    __device__ __forceinline__ bool bad() const { return false; }
};

struct FastMath {
    static constexpr bool kZeroTest = false;  // a zero divisor is out of range: the solve is done again
    using Rec = double;  // the correctly rounded reciprocal of a divisor
    // smallest (2 |hi| + (lo != 0)) - 1 and largest 2 |hi| of the numerators; smallest and largest
    // high word of the divisors and radicands.  A zero numerator passes (its entry wraps to the
    // largest unsigned value); zero, negative, infinite and NaN divisors do not.
    unsigned nmin = 0xffffffffu, nmax = 0u;
    unsigned dmin = 0xffffffffu, dmax = 0u;

    __host__ __device__ static constexpr unsigned hiword(int e) { return (unsigned)(1023 + e) << 20; }  // of 2^e
    __device__ __forceinline__ void numer(double a) {
        const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
        const unsigned u = hi + hi + min(lo, 1u);
        nmin = min(nmin, u - 1u);
        nmax = max(nmax, u);
    }
    __device__ __forceinline__ void denom(double b) {
        const unsigned hi = (unsigned)__double2hiint(b);
        dmin = min(dmin, hi);
        dmax = max(dmax, hi);
    }
    // numerators zero or in [2^-700, 2^700], divisors and radicands in [2^-200, 2^200]: every
    // quotient, remainder and correction is then zero or a normal number
    __device__ __forceinline__ bool bad() const {
        return nmin < 2u * hiword(-700) || nmax > 2u * hiword(700) || dmin < hiword(-200) || dmax > hiword(200);
    }

    __device__ __forceinline__ static double seed(double b) {
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
        return y;
    }
    // RN(1/b) from an approximation y >= about 1/b within an ulp
    __device__ __forceinline__ static double sharpen(double b, double y) { return __fma_rn(__fma_rn(-b, y, 1.0), y, y); }
    __device__ __forceinline__ Rec rec(double b) {
        denom(b);
        const double y = seed(b);
        const double e = __fma_rn(-b, y, 1.0);
        return sharpen(b, __fma_ru(__fma_rn(e, e, e), y, y));  // y (1 + e + e^2)
    }
    __device__ __forceinline__ static double quot(double a, double b, Rec y) {  // without a look at a
        const double q = a * y;
        return __fma_rn(-__fma_rn(b, q, -a), y, q);
    }
    __device__ __forceinline__ double div(double a, double b, Rec y) {
        numer(a);
        return quot(a, b, y);
    }
    __device__ __forceinline__ double inv(double b) { return rec(b); }
    // the root of x, and z = 1 / sqrt(x) to within an ulp
    __device__ __forceinline__ double root_z(double x, double &z) {
        denom(x);
        double y;
        asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
        double g = x * y;
        const double t = __fma_rn(-g, y, 1.0);
        const double s = t * __fma_rn(0.375, t, 0.5);  // (1 - t)^(-1/2) = 1 + t/2 + 3 t^2/8 + ...
        g = __fma_rd(g, s, g);
        z = __fma_rn(y, s, y);
        return __fma_rn(0.5 * __fma_rn(-g, g, x), z, g);
    }
    __device__ __forceinline__ double root(double x) {
        double z;
        return root_z(x, z);
    }
    // s = sqrt(x) and RN(1/s)
    __device__ __forceinline__ double root(double x, Rec &is) {
        double z;
        const double s = root_z(x, z);
        is = sharpen(s, __fma_ru(__fma_rn(-s, z, 1.0), z, z));
        return s;
    }
    __device__ __forceinline__ double inv_root(double x) {
        Rec is;
        root(x, is);
        return is;
    }
};

}  // namespace dg
