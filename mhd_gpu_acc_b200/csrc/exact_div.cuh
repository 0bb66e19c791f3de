// exact_div.cuh -- correctly rounded FP64 quotients and square roots without a
// branch per operation.
//
// The FP64 sweeps are bounded by latency: about 33 divisions and 6 square roots
// per cell and sweep, and the compiler's division and root each end in a branch
// to their slow path, which keeps one chain from overlapping the next.  Here a
// group of independent quotients is formed as straight-line code, with one
// branch for the group to the plain operators when an operand lies outside the
// range in which the short form is exact.
//
// Method (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990, and its restatement in
// Muller et al., "Handbook of Floating-Point Arithmetic", ch. 4): from y1 with
// 1 - b y1 = e1 known exactly (one FMA), y = y1 + e1 y1 is the correctly rounded
// reciprocal unless b's significand is all ones (such b count as out of range);
// t = a y1, q = t + e1 t is within one ulp of a / b, its residual s = a - b q is
// exact, and q + s y is the correctly rounded quotient.  The first y1 is the
// hardware's reciprocal approximation (20 bits, rcp.approx.ftz.f64) with one
// third-order step.  The root is the same iteration on 1 / sqrt(x): s + h (x - s^2)
// with h = 1 / (2 sqrt(x)).  tests/exact_div_check.cu compares both with the
// operators on random operands and on the hardest roundings.
//
// Ranges: |b| in [2^-480, 2^60), numerators zero or in [2^-960, 2^540) by magnitude,
// roots of +0 or [2^-900, 2^900): then quotients lie in (2^-1021, 2^1021), so that none
// is subnormal or overflows, and the residuals, multiples of 2^-1064, are exact.
// tests/exact_range_check.cu draws both operands from all of these ranges.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define XD_HD __host__ __device__ __forceinline__
#else
#define XD_HD inline
#endif

namespace mhd {
namespace exact {

XD_HD unsigned hi_word(double a) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(a);
#else
    std::uint64_t b;
    std::memcpy(&b, &a, 8);
    return (unsigned)(b >> 32);
#endif
}
XD_HD unsigned lo_word(double a) {
#ifdef __CUDA_ARCH__
    return (unsigned)__double2loint(a);
#else
    std::uint64_t b;
    std::memcpy(&b, &a, 8);
    return (unsigned)b;
#endif
}

// Whether |a| lies outside [2^LO, 2^HI); twice the high word drops the sign.
template <int LO, int HI>
XD_HD bool xd_out(double a) {
    constexpr unsigned lo = (unsigned)(1023 + LO) << 21, span = (unsigned)(HI - LO) << 21;
    const unsigned h = hi_word(a);
    return (h + h) - lo >= span;
}
XD_HD bool out_den(double b) { return xd_out<-480, 60>(b) | (lo_word(b) == 0xffffffffu); }
XD_HD bool out_num(double a) { return (a != 0.0) & xd_out<-960, 540>(a); }
// -0, negative and NaN radicands are out of range too (the unsigned difference)
XD_HD bool out_rad(double x) {
    constexpr unsigned lo = (unsigned)(1023 - 900) << 20, span = 1800u << 20;
    const unsigned h = hi_word(x);
    return (h - lo >= span) & ((h | lo_word(x)) != 0u);
}

// The approximations that the iterations start from (a stand-in of the same
// width on the host).
XD_HD double rcp_seed(double b) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    return y;
#else
    double y = 1.0 / b;
    std::uint64_t u;
    std::memcpy(&u, &y, 8);
    u &= 0xffffffff00000000ull;
    std::memcpy(&y, &u, 8);
    return y;
#endif
}
XD_HD double rsqrt_seed(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
#else
    double y = 1.0 / std::sqrt(x);
    std::uint64_t u;
    std::memcpy(&u, &y, 8);
    u &= 0xffffffff00000000ull;
    std::memcpy(&y, &u, 8);
    return y;
#endif
}

// A denominator's reciprocal: y correctly rounded, y1 near it with 1 - b y1 = e1.
struct Recip {
    double b, y1, e1, y;
};
XD_HD Recip recip(double b) {
    Recip r;
    r.b = b;
    const double y0 = rcp_seed(b), e = fma(-b, y0, 1.0);
    r.y1 = fma(y0, fma(e, e, e), y0);
    r.e1 = fma(-b, r.y1, 1.0);
    r.y = fma(r.e1, r.y1, r.y1);
    return r;
}
// From a correctly rounded reciprocal y of b.
XD_HD Recip recip_of(double b, double y) { return Recip{b, y, fma(-b, y, 1.0), y}; }

// a / r.b, correctly rounded, for operands in range; a zero numerator keeps the
// sign that the division gives it.
XD_HD double quot(double a, const Recip& r) {
    const double t = a * r.y1, q = fma(t, r.e1, t), s = fma(-r.b, q, a);
    const double w = fma(s, r.y, q);
    return a == 0.0 ? t : w;
}
// The same for a >= 0 over a positive denominator (no signed zero to keep).
XD_HD double quot_pos(double a, const Recip& r) {
    const double t = a * r.y1, q = fma(t, r.e1, t), s = fma(-r.b, q, a);
    return fma(s, r.y, q);
}

// sqrt(x), correctly rounded, for x in range.
XD_HD double root(double x) {
    const double y0 = rsqrt_seed(x), g0 = x * y0, e = fma(-g0, y0, 1.0);
    const double y1 = fma(y0 * e, fma(e, 0.375, 0.5), y0);
    const double h = 0.5 * y1, g1 = x * y1;
    const double g2 = fma(fma(-g1, g1, x), h, g1);
    const double g3 = fma(fma(-g2, g2, x), h, g2);
    return x == 0.0 ? x : g3;
}

// y[i] = 1 / b[i], correctly rounded.
template <int N>
XD_HD void reciprocals(const double* b, double* y) {
    bool bad = false;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        y[i] = recip(b[i]).y;
        bad |= out_den(b[i]);
    }
    if (bad) {
#pragma unroll
        for (int i = 0; i < N; ++i) y[i] = 1.0 / b[i];
    }
}

}  // namespace exact
}  // namespace mhd
