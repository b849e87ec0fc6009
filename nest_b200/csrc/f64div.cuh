// Correctly rounded FP64 division and square root without slow-path branches,
// for the FP64 plain form (sm_100a; every fused multiply-add below is an
// explicit fma(), so the units' -fmad=false does not matter here).
//
// The IEEE division and square root that nvcc emits for `a / b` and `sqrt(x)`
// carry a rarely taken slow path each, and a stage has 20 divisions and five
// square roots a cell: their branches, not the FP64 arithmetic, held the
// kernels back.  The forms here have no branch and no rounding test.  They
// return the IEEE result whenever the operands lie in a safe range; a kernel
// accumulates the range tests of everything that reaches an output in an
// F64Range and, where one fails, repeats the work with the IEEE operations
// before anything is stored.
//
// Division a / b (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990; J.-M. Muller
// et al., Handbook of Floating-Point Arithmetic, 2nd ed., 2018, ch. 4):
//   * y = recip_f64(b): from the hardware approximation y0 (measured over every
//     high word: |1 - b y0| < 2^-19.9) three Newton-Raphson steps
//     y <- y + y (1 - b y).  The second leaves 1/b to 2^-79 and its rounding; it
//     rounds up, so that y is 1/b at least (to 2^-79) and less than an ulp above.
//     The last one's residual e is exact, |e| <= m_b 2^-53 (m_b in [1, 2) the
//     significand of b), so y is the rounding of (1/b)(1 - e^2).  The reciprocal of
//     b = 2 - ulp lies next to a midpoint, 2^-106 above it, the nearest of all:
//     rounded to nearest the second step fell below it, and the last was a tie that
//     stayed there.  From above it ends at RN(1/b), and so does b = 2 - 2 ulp.
//     One y serves every quotient by b.
//   * q0 = a y, r = b q0 - a, q = q0 - r y (quot_f64).  With eps the relative
//     error of y, q is the rounding of a/b + (a/b - q0) eps.  A quotient of
//     two doubles stays at least ulp(q) 2^-53 / m_b away from every midpoint
//     of two doubles, and |eps| <= m_b 2^-54 + m_b^2 2^-106.  Next to a midpoint
//     |a/b - q0| is half an ulp, or one and a half if q0 is not a faithful
//     rounding.  Half an ulp: the perturbation is smaller than the distance
//     where (m_b / 2)^2 (1 + m_b 2^-52) < 1, for all but the two divisors above, whose
//     y = RN(1/b) has an eps of 2^-53 - 2^-106 and 2^-104.
//     One and a half: q0 = RN(a y) can only be that far off where a's
//     significand exceeds 2 - 5 2^-52 and b's is larger still, and all
//     those quotients lie next to a double, not next to a midpoint.  So q =
//     RN(a / b).
//   * r = b q0 - a rather than a - b q0 keeps the sign of a zero quotient:
//     with b > 0, a = -0 gives r = +0 and q = q0 - 0 = -0.
// Square root (Markstein, as above, and Goldschmidt's iteration: P. Markstein,
// "Software division and square root using Goldschmidt's algorithms", RNC6,
// 2004): from the hardware approximation y0 (measured: |1 - x y0^2| < 2^-19.0)
// g ~ s = sqrt(x) and h ~ 1 / (2 s) together, g <- g + g r, h <- h + h r with
// r = 1/2 - g h (2^-39), then h once more, with relative error eta, then twice
// g <- g + (x - g^2) h.  The first of these leaves g within half an ulp (and a few 2^-26
// of one) of s; the second has an exact residual and rounds s - d^2 / (2 s) + d eta
// (d = s - g).  With s in [1, 2) and ulp = 2^-52, eta is the rounding of h and half the
// rounding of g, at most (s + 1/s) ulp / 4, so next to a midpoint, where |d| is half an
// ulp, at most ulp^2 s / 8 is added to s and ulp^2 (s + 2/s) / 8 taken from it.  A
// midpoint m below s has s - m >= 7 ulp^2 / (8 s) (in units of ulp^2 / 4, m^2 is 1
// modulo 8 and x a multiple of 8), more than is taken; one above s has m - s >= 9 ulp^2 /
// (8 s), more than is added, but for x = 1 + ulp and x = 4 - 2 ulp, where it is ulp^2 /
// (8 s).  sqrt_f64's steps depend on x alone, and tests/test_gpu_div.py runs it on these
// two; sqrt_quot_f64's depend on the quotient's operands too, so the kernels do not
// keep its root of these two (F64Range::root).
#pragma once

#include <cuda_runtime.h>

namespace nestb {

__device__ __forceinline__ double recip_f64(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = fma(y, fma(-b, y, 1.0), y);
    y = __fma_ru(y, fma(-b, y, 1.0), y);
    return fma(y, fma(-b, y, 1.0), y);
}

// RN(a / b) for y = recip_f64(b), in range.
__device__ __forceinline__ double quot_f64(double a, double b, double y) {
    const double q = a * y;
    return fma(-fma(b, q, -a), y, q);
}

// RN(sqrt(x)), in range.
__device__ __forceinline__ double sqrt_f64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double h = 0.5 * y, g = x * y;
    const double r = fma(-g, h, 0.5);
    h = fma(h, r, h);
    g = fma(g, r, g);
    h = fma(h, fma(-g, h, 0.5), h);
    g = fma(fma(-g, g, x), h, g);
    return fma(fma(-g, g, x), h, g);
}

// RN(sqrt(q)) with q = RN(a / b), in range and not one of the two arguments above, and q: the same steps as recip_f64, quot_f64 and sqrt_f64,
// with the square root's first approximation taken from a quotient of 2^-39 relative
// error, so that it runs beside the exact quotient instead of after it (the second
// Newton-Raphson step of h and everything after it use the exact q).
__device__ __forceinline__ double sqrt_quot_f64(double a, double b, double& q) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = fma(y, fma(-b, y, 1.0), y);
    const double t = a * y, t2 = t + t;
    double h;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(h) : "d"(t));
    h *= 0.5;
    h = fma(h, fma(-(t2 * h), h, 0.5), h);  // 1 / (2 sqrt(q)) to 2^-39
    y = __fma_ru(y, fma(-b, y, 1.0), y);
    y = fma(y, fma(-b, y, 1.0), y);
    q = quot_f64(a, b, y);
    double g = (q + q) * h;
    h = fma(h, fma(-g, h, 0.5), h);
    g = fma(fma(-g, g, q), h, g);
    return fma(fma(-g, g, q), h, g);
}

// Whether q = quot_f64(a, b, recip_f64(b)), b > 0, lies where the argument above
// holds on its own: b in [2^-960, 2^961), and a = 0 or |a| and |q| in
// [2^-959, 2^961).  (The kernels use the cheaper F64Range, which is narrower.)
__device__ __forceinline__ bool f64_exp_safe(double x, unsigned lo) {
    return (((unsigned)__double2hiint(x) >> 20) & 0x7ffu) - lo < 1984u - lo;
}
__device__ __forceinline__ bool quot_in_range(double a, double b, double q) {
    return f64_exp_safe(b, 63) && (a == 0.0 || (f64_exp_safe(a, 64) && f64_exp_safe(q, 64)));
}

// Range tests, accumulated over a group of operations and read once.
//   pos(x): x in [2^-128, 2^128).  Adding a constant to the high word moves
//     that range of exponents to the top 16th of the exponent field and, for
//     a positive x, sets the sign bit: the AND over all x keeps the top four
//     bits set only if every x passes (two integer operations each).
//   num(a): a = 0 or |a| >= 2^-800.  Twice the high word, less one where the
//     low word is 0, is 0xffffffff for a zero, below 2 for a subnormal, and
//     orders by exponent otherwise; the minimum is kept.
// With b in [2^-129, 2^192) and |a| < 2^880 a quotient whose numerator passes
// num() is 0 or normal, nothing overflows, and b q - a is a multiple of
// 2^-1074, so the residual above is exact.
struct F64Range {
    unsigned all = 0xffffffffu, low = 0xffffffffu;
    __device__ __forceinline__ void pos(double x) {
        all &= (unsigned)__double2hiint(x) + ((897u << 20) ^ 0x80000000u);
    }
    __device__ __forceinline__ void num(double a) {
        unsigned k;  // 2 hi + (lo != 0) - 1: the first addition carries where lo != 0
        asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %1, 0xffffffff;\n\taddc.u32 %0, %2, 0xffffffff;\n\t}"
            : "=r"(k) : "r"(__double2loint(a)), "r"(2u * (unsigned)__double2hiint(a)));
        low = min(low, k);
    }
    // root(q): q is not (1 + ulp) 4^k or (4 - 2 ulp) 4^k.  (Nor twice those: the
    // fraction field alone is tested, for 1 and for all ones.)
    __device__ __forceinline__ void root(double q) {
        const unsigned hi = (unsigned)__double2hiint(q), lo = (unsigned)__double2loint(q);
        const unsigned away = ((lo + 1u) & ~2u) | ((hi + (lo >> 31)) & 0xfffffu);
        low = away == 0u ? 0u : low;
    }
    __device__ __forceinline__ bool ok() const { return all >= 0xf0000000u && low >= (223u << 21); }
};

// Arithmetic policies: the IEEE division and square root, or the branch-free
// ones with their range tests.  Both give the same values wherever ok() holds
// in the end.
struct ArithIeee {
    static constexpr bool checked = false;
    struct Recip { double b; };
    __device__ __forceinline__ Recip recip(double b) const { return { b }; }
    __device__ __forceinline__ double quot(double a, const Recip& r) const { return a / r.b; }
    __device__ __forceinline__ double root(double x) const { return sqrt(x); }
    __device__ __forceinline__ double inverse(double b) const { return 1.0 / b; }
    __device__ __forceinline__ double half(double w, double h, double s) const { return w + h * s; }
    __device__ __forceinline__ void pos(double) {}
    __device__ __forceinline__ void num(double) {}
    __device__ __forceinline__ bool ok() const { return true; }
};
struct ArithFast {
    static constexpr bool checked = true;
    struct Recip { double b, y; };
    F64Range r;
    __device__ __forceinline__ Recip recip(double b) const { return { b, recip_f64(b) }; }
    __device__ __forceinline__ double quot(double a, const Recip& q) const { return quot_f64(a, q.b, q.y); }
    __device__ __forceinline__ double root(double x) const { return sqrt_f64(x); }
    // 1 / b to within a rounding (recip_f64), for terms that no branch compares
    __device__ __forceinline__ double inverse(double b) const { return recip_f64(b); }
    // sqrt(a / b)
    __device__ __forceinline__ double root_quot(double a, double b) { return root(quot(a, recip(b))); }
    // h = +-1/2: h s is exact (slopes in range are multiples of 2^-1000), so the
    // fused form rounds the same sum
    __device__ __forceinline__ double half(double w, double h, double s) const { return fma(h, s, w); }
    __device__ __forceinline__ void pos(double x) { r.pos(x); }
    __device__ __forceinline__ void num(double a) { r.num(a); }
    __device__ __forceinline__ bool ok() const { return r.ok(); }
};
// The same with the square root's approximation beside the quotient: a shorter chain for
// a multiplication and a range test more.  For the resident 1D loop, which the chain
// bounds (us a step at 100 / 1024 cells 1.356 -> 1.333, 1.980 -> 1.956); the kernels of many
// warps are faster without (1D step at 200003 cells 10.53 -> 10.26, reverse step at
// 65536 13.35 -> 13.07, pipeline of 400 cells 6.03 -> 5.95).
struct ArithChain : ArithFast {
    __device__ __forceinline__ double root_quot(double a, double b) {
        double q;
        const double s = sqrt_quot_f64(a, b, q);
        r.root(q);
        return s;
    }
};

// RN(a / b) for one quotient by a divisor that changes.
__device__ __forceinline__ double div_rn(double a, double b) {
    F64Range r;
    r.pos(b);
    r.pos(a);
    const double q = quot_f64(a, b, recip_f64(b));
    return r.ok() ? q : a / b;
}

}  // namespace nestb
