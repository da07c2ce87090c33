// FP64 quotients that round exactly like IEEE division, without its branches.
//
// The plain form's WENO weights are chains of divisions by positive numbers
// of moderate size.  The compiler's division tests its operands and branches
// on every call, so neighbouring quotients cannot overlap and the FP64 pipe
// waits on their latency (WENO5: 6 divisions a point).  Here the operand
// test is made once for a group of divisors, the quotients are straight
// line code, and divisions by the same number share its reciprocal.
//
// Method: Newton's series for the reciprocal, then Markstein's quotient
// correction (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).
//   y = y0 (1 + e + e^2 + e^3), e = 1 - b y0, from the hardware's
//   approximation y0 (of b's high word: |e| <= 2^-18, tested over all significands
//   of 20 bits, tests/test_div64_gpu.py): |y - 1/b| <= (1/2 + 2^-18) ulp;
//   q0 = RN(a y), r = a - b q0, q = RN(q0 + r y).
// Why q = RN(a / b) when b's significand B is at most 2 - 2^-15 and neither
// a y nor r leaves the normal range.  Let A be a's significand, h = 1/2 + 2^-18.
// q0 is off by e0 <= 1/2 + A h ulp when A < B, else by less than 1 ulp.
//  * |e0| < 1 ulp: r is exact, an integer multiple of ulp(b) ulp(q0).  With
//    k = 2^52 B, a quotient next to the midpoint q0 + 1/2 ulp has
//    |r| >= (k + 1) / 2 such units above it (or <= (k - 1) / 2 below), so r y
//    falls on the right side if y's relative error is below 1/(k + 1); it is
//    at most h 2^-53 B, and h B^2 < 2 for this B.
//  * 1 <= |e0|: then A < B <= 2 - 2^-15 and |e0| <= 1/2 + A h < 3/2 - 2^-17,
//    at least 2^-17 ulp from either midpoint, while the errors of r (one unit,
//    2^-52 ulp) and of r y (2^-51 ulp) are far smaller.
#pragma once

namespace mth {

// Whether b may be a divisor of div_by below: (hi word) significand at most
// 2 - 2^-15.  Adding 2^-15 then leaves the exponent bits alone; returns a word
// whose bit 20 is set otherwise.
__device__ __forceinline__ int div_edge(double b) {
  const int hi = __double2hiint(b);
  return (hi + 0x20) ^ hi;
}
constexpr int kDivEdge = 0x100000;

// The reciprocal of a normal b as div_by needs it.
__device__ __forceinline__ double div_rcp(double b) {
  double y0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
  const double e = __fma_rn(-b, y0, 1.0);
  const double p = __fma_rn(e, __fma_rn(e, e, e), e);
  return __fma_rn(y0, p, y0);
}

// RN(a / b), y = div_rcp(b).
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}

static __device__ __noinline__ double div_ieee(double a, double b) { return a / b; }

// Quotients by one divisor, x / d, for many x of any size, all rounded like
// IEEE division.  d from 2^-100 to 2^100 (but the edge above): RN(1 / d) once (the
// bound above holds with h = 1/2), then three operations for an x of 2^-900 to
// 2^900, none for a zero.  Any other x or d (negative, zero, infinite, NaN)
// divides, out of line.
struct Divisor {
  double d, y;
  unsigned span;
  __device__ __forceinline__ explicit Divisor(double dd) : d(dd), y(1.0 / dd) {
    const bool ok = dd >= 0x1p-100 && dd <= 0x1p100 && !(div_edge(dd) & kDivEdge);
    span = ok ? 1800u << 20 : 0u;
  }
  __device__ __forceinline__ double operator()(double x) const {
    const unsigned hi = (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
    if (hi - (123u << 20) < span) return div_by(x, d, y);
    return x == 0.0 && span ? x : div_ieee(x, d);
  }
};

// 1/x and 1/sqrt(x) for the mixed form, without the branches of the library's
// division and rsqrt, by Newton's series from the hardware's approximations:
// of a normal x (rsqrt64: a positive one) whose reciprocal is normal too, to
// 0.51 and 1.2 ulp (x y0^2 = 1 - e, |e| < 2^-18, for the root y = y0 (1 + e/2 + 3/8 e^2
// + ...), whose e^3 term is below 2^-55).  An infinite, zero or subnormal x gives
// NaN, a reciprocal below 2^-1022 gives 0: callers keep their operands away from
// there.  The recoveries are chains of them at 40-48% of the FP64 pipe, bound by
// the chains' latency.
__device__ __forceinline__ double rcp64(double x) { return div_rcp(x); }
__device__ __forceinline__ double rsqrt64(double x) {
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
  const double e = fma(-(x * y0), y0, 1.0);
  return fma(y0 * e, fma(0.375, e, 0.5), y0);
}

}  // namespace mth
