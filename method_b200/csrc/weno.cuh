// WENO3 / WENO5 point reconstructions.
//
// `Weno3Point` / `Weno5Point` evaluate the same expressions, in the same order,
// as the reference's generated point kernels
// (Project/CPU/Src/wenoUpwinds.cc:5-33 and 36-83): smoothness indicators
// accumulated term by term from zero, alpha_k = d_k / (1e-16 + beta_k^2),
// weights by division by the alpha sum, stencils accumulated term by term.
// Compiled without FMA contraction (-fmad=false) they are bit-identical to the
// reference's x86-64 build.  The downwind value at a face is the same
// function applied to the mirrored stencil (Project/CPU/Src/weno.cc:145-164,
// 208-228), so only the upwind form exists here.
//
// `weno3_fast2` / `weno5_fast2` are the FP32 forms of the mixed-precision
// path: the same Jiang-Shu weights, regrouped for FMA, with approximate
// reciprocals, evaluating the upwind and downwind sides of a face together.
#pragma once
#include "div64.cuh"

namespace mth {

// The divisions of a point (alpha_k and w_k) as div64.cuh's branch-free
// quotients: one operand test per point, the three alpha_k side by side, the
// w_k on one reciprocal of the alpha sum.  Same bits as IEEE divisions; a
// point whose operands fail the test (an indicator above 2^448, NaN, or a
// divisor's significand within 2^-15 of 2) takes them, out of line.  A sum
// that the reference starts from zero starts from its first term here: for
// an indicator that term is never -0, and for a candidate stencil only the
// sign of a zero face value could change, which the + 0.0 restores.
//
// Bound by the FP64 pipe and issue: OT 1024^2 WENO5, grouped tile, 0.510 -> 0.44
// ms per launch with these quotients and 0.41 with the faces scaled once
// (fvs2d.cuh); 100 -> 73 M warp instructions per 512^2 launch.
constexpr unsigned kWenoTop = 0x77F00000u;  // high word of 2^896

static __device__ __noinline__ double weno3_ieee(double q0, double q1, double s0, double s1) {
  const double a0 = 0.3333333333333333 / q0, a1 = 0.6666666666666666 / q1;
  const double asum = a0 + a1;
  const double w0 = a0 / asum, w1 = a1 / asum;
  return (w0 * s0 + w1 * s1);
}

static __device__ __noinline__ double weno5_ieee(double q0, double q1, double q2, double s0,
                                                 double s1, double s2) {
  const double a0 = 0.1 / q0, a1 = 0.6 / q1, a2 = 0.3 / q2;
  const double asum = a0 + a1 + a2;
  const double w0 = a0 / asum, w1 = a1 / asum, w2 = a2 / asum;
  return (w0 * s0 + w1 * s1 + w2 * s2);
}

// The candidate stencils and eps + beta_k^2 of one point.
struct Weno3Point {
  double q0, q1, s0, s1;
  __device__ __forceinline__ Weno3Point(double v0, double v1, double v2) {
    const double eps = 1e-16;
    double b0 = 1.0 * v1 * v1;
    b0 += -2.0 * v0 * v1;
    b0 += 1.0 * v0 * v0;
    double b1 = 1.0 * v2 * v2;
    b1 += -2.0 * v1 * v2;
    b1 += 1.0 * v1 * v1;
    q0 = eps + b0 * b0;
    q1 = eps + b1 * b1;
    s0 = 1.5 * v1;
    s0 += -0.5 * v0;
    s1 = 0.5 * v2;
    s1 += 0.5 * v1;
  }
  // The reconstruction; `edge` and `top` collect the operand test.
  __device__ __forceinline__ double fast(int& edge, unsigned& top) const {
    const double a0 = div_by(0.3333333333333333, q0, div_rcp(q0));
    const double a1 = div_by(0.6666666666666666, q1, div_rcp(q1));
    const double asum = a0 + a1;
    const double y = div_rcp(asum);
    const double w0 = div_by(a0, asum, y), w1 = div_by(a1, asum, y);
    edge |= div_edge(q0) | div_edge(q1) | div_edge(asum);
    top = max(top, max((unsigned)__double2hiint(q0), (unsigned)__double2hiint(q1)));
    return (w0 * s0 + w1 * s1);
  }
  __device__ __forceinline__ double ieee() const { return weno3_ieee(q0, q1, s0, s1); }
};

struct Weno5Point {
  double q0, q1, q2, s0, s1, s2;
  __device__ __forceinline__ Weno5Point(double v0, double v1, double v2, double v3, double v4) {
    const double eps = 1e-16;
    double b0 = 3.3333333333333335 * v2 * v2;
    b0 += -10.333333333333334 * v1 * v2;
    b0 += 8.333333333333334 * v1 * v1;
    b0 += 3.6666666666666665 * v0 * v2;
    b0 += -6.333333333333333 * v0 * v1;
    b0 += 1.3333333333333333 * v0 * v0;
    double b1 = 1.3333333333333333 * v3 * v3;
    b1 += -4.333333333333333 * v2 * v3;
    b1 += 4.333333333333333 * v2 * v2;
    b1 += 1.6666666666666667 * v1 * v3;
    b1 += -4.333333333333333 * v1 * v2;
    b1 += 1.3333333333333333 * v1 * v1;
    double b2 = 1.3333333333333333 * v4 * v4;
    b2 += -6.333333333333333 * v3 * v4;
    b2 += 8.333333333333334 * v3 * v3;
    b2 += 3.6666666666666665 * v2 * v4;
    b2 += -10.333333333333334 * v2 * v3;
    b2 += 3.3333333333333335 * v2 * v2;
    q0 = eps + b0 * b0;
    q1 = eps + b1 * b1;
    q2 = eps + b2 * b2;
    s0 = 1.8333333333333333 * v2;
    s0 += -1.1666666666666667 * v1;
    s0 += 0.3333333333333333 * v0;
    s1 = 0.3333333333333333 * v3;
    s1 += 0.8333333333333334 * v2;
    s1 += -0.16666666666666666 * v1;
    s2 = -0.16666666666666666 * v4;
    s2 += 0.8333333333333334 * v3;
    s2 += 0.3333333333333333 * v2;
  }
  __device__ __forceinline__ double fast(int& edge, unsigned& top) const {
    const double a0 = div_by(0.1, q0, div_rcp(q0));
    const double a1 = div_by(0.6, q1, div_rcp(q1));
    const double a2 = div_by(0.3, q2, div_rcp(q2));
    const double asum = a0 + a1 + a2;
    const double y = div_rcp(asum);
    const double w0 = div_by(a0, asum, y), w1 = div_by(a1, asum, y), w2 = div_by(a2, asum, y);
    edge |= div_edge(q0) | div_edge(q1) | div_edge(q2) | div_edge(asum);
    top = max(top, max(max((unsigned)__double2hiint(q0), (unsigned)__double2hiint(q1)),
                       (unsigned)__double2hiint(q2)));
    return (w0 * s0 + w1 * s1 + w2 * s2);
  }
  __device__ __forceinline__ double ieee() const { return weno5_ieee(q0, q1, q2, s0, s1, s2); }
};

// The point of order ORDER on v[0], v[stride], ...
template <int ORDER>
__device__ __forceinline__ auto weno_load(const double* v, long long stride) {
  if constexpr (ORDER == 3)
    return Weno3Point(v[0], v[stride], v[2 * stride]);
  else
    return Weno5Point(v[0], v[stride], v[2 * stride], v[3 * stride], v[4 * stride]);
}

__device__ __forceinline__ bool weno_operands_ok(int edge, unsigned top) {
  return top < kWenoTop && !(edge & kDivEdge);
}

// Both points of a face again, from memory, with IEEE divisions.
template <int ORDER>
__device__ __noinline__ double weno_face_ieee(const double* p, const double* m, long long stride) {
  return weno_load<ORDER>(p, stride).ieee() + weno_load<ORDER>(m, -stride).ieee() + 0.0;
}

// A face of order 3 or 5: the upwind point of f+ at p, p + stride, ... plus
// the downwind point of f- at m, m - stride, ....
// PAIR: one operand test after both points, so that their chains overlap; a
// face that fails it starts over from memory, so nothing is kept for that.
// The few warps of a small grid gain by it (KH 64 x 128 step, one-pass tile:
// 0.077 against 0.080 ms).  The grouped tile, with 64 registers and 32 warps on
// an SM, is the faster with one point after the other (OT 1024^2 step 1.51
// against 1.525 ms).
template <int ORDER, bool PAIR>
__device__ __forceinline__ double weno_face_exact(const double* p, const double* m,
                                                  long long stride) {
  int edge = 0;
  unsigned top = 0;
  const auto up = weno_load<ORDER>(p, stride);
  double u = up.fast(edge, top);
  if constexpr (!PAIR) {
    if (!weno_operands_ok(edge, top)) u = up.ieee();
    edge = 0;
    top = 0;
  }
  const auto dn = weno_load<ORDER>(m, -stride);
  double d = dn.fast(edge, top);
  if (!weno_operands_ok(edge, top)) {
    if constexpr (PAIR) return weno_face_ieee<ORDER>(p, m, stride);
    d = dn.ieee();
  }
  return u + d + 0.0;  // + 0.0: a zero face value is +0, as the reference's sums from zero give
}

// FP32 forms: two reconstructions at once in FP32x2 arithmetic (sm_100
// __ffma2_rn / __fadd2_rn / __fmul2_rn: one instruction for both lanes, each
// rounded as the scalar operation) -- two variables of one side of a face, or
// the upwind (.x) and downwind (.y) sides of one variable.
//
// In first differences d_k = v_{k+1} - v_k and second ones t_k = d_{k+1} - d_k
// the Jiang-Shu indicators (times 4) are 13/3 t^2 + u^2 with u_0 = t_0 + 2 d_1,
// u_1 = d_1 + d_2, u_2 = t_2 - 2 d_2, and the face value is v_2 plus the weighted
// corrections d_1/2 + t_0/3, d_2/2 - t_1/6, d_2/2 - t_2/6.  With q_k = eps +
// beta_k^2 (eps times 16) the weights (c_k / q_k) / sum_j (c_j / q_j), c = 1 : 6 : 3,
// equal c_k P_k / sum_j c_j P_j with P_k the product of the other two q, so only
// the final normalisation divides.  The q are first scaled by the power of two
// that brings their sum into [2^30, 2^31) (exponent bits only, exact): the
// products then neither overflow nor fall out of the normal range, for
// jumps up to where beta^2 itself overflows, so an approximate reciprocal
// without subnormal handling serves.  (WENO3's two weights are normalised before
// they meet the differences, which serves as well.)
// 47 instructions a pair of points, 59 before in the form with separate
// stencil sums and maximum-based scaling.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

__device__ __forceinline__ float rcp_normal(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float2 rcp2(float2 q) {
  return make_float2(rcp_normal(q.x), rcp_normal(q.y));
}

// 2^(30 - floor(log2 s)) for a normal s of at least 2^-90, from the exponent bits.
__device__ __forceinline__ float pow2_scale(float s) {
  return __uint_as_float(0x8E000000u - (__float_as_uint(s) & 0x7F800000u));
}

__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  return __ffma2_rn(f2(-1.0f), b, a);
}

// v_1 + (q_1 / Q) d_0 / 2 + (q_0 / Q) d_1, Q = q_1 + 2 q_0: linear weights 1 : 2.
__device__ __forceinline__ float2 weno3_fast2(float2 v0, float2 v1, float2 v2) {
  const float2 d0 = sub2(v1, v0), d1 = sub2(v2, v1);
  const float2 b0 = __fmul2_rn(d0, d0), b1 = __fmul2_rn(d1, d1);
  const float2 q0 = __ffma2_rn(b0, b0, f2(1e-16f)), q1 = __ffma2_rn(b1, b1, f2(1e-16f));
  const float2 r = rcp2(__ffma2_rn(f2(2.0f), q0, q1));
  return __ffma2_rn(__fmul2_rn(q1, r), __fmul2_rn(f2(0.5f), d0),
                    __ffma2_rn(__fmul2_rn(q0, r), d1, v1));
}

__device__ __forceinline__ float2 weno5_fast2(float2 v0, float2 v1, float2 v2, float2 v3,
                                              float2 v4) {
  const float2 d0 = sub2(v1, v0), d1 = sub2(v2, v1), d2 = sub2(v3, v2), d3 = sub2(v4, v3);
  const float2 t0 = sub2(d1, d0), t1 = sub2(d2, d1), t2 = sub2(d3, d2);
  const float2 u0 = __ffma2_rn(f2(2.0f), d1, t0);
  const float2 u1 = __fadd2_rn(d1, d2);
  const float2 u2 = __ffma2_rn(f2(-2.0f), d2, t2);
  const float2 c13 = f2(13.0f / 3.0f);
  const float2 b0 = __ffma2_rn(__fmul2_rn(c13, t0), t0, __fmul2_rn(u0, u0));
  const float2 b1 = __ffma2_rn(__fmul2_rn(c13, t1), t1, __fmul2_rn(u1, u1));
  const float2 b2 = __ffma2_rn(__fmul2_rn(c13, t2), t2, __fmul2_rn(u2, u2));
  float2 q0 = __ffma2_rn(b0, b0, f2(16e-16f));
  float2 q1 = __ffma2_rn(b1, b1, f2(16e-16f));
  float2 q2 = __ffma2_rn(b2, b2, f2(16e-16f));
  const float2 qs = __fadd2_rn(__fadd2_rn(q0, q1), q2);
  const float2 sc = make_float2(pow2_scale(qs.x), pow2_scale(qs.y));
  q0 = __fmul2_rn(q0, sc);
  q1 = __fmul2_rn(q1, sc);
  q2 = __fmul2_rn(q2, sc);
  const float2 p0 = __fmul2_rn(q1, q2), p1 = __fmul2_rn(q0, q2), p2 = __fmul2_rn(q0, q1);
  // the corrections times 1, 6, 3
  const float2 e0 = __ffma2_rn(f2(1.0f / 3.0f), t0, __fmul2_rn(f2(0.5f), d1));
  const float2 e1 = __ffma2_rn(f2(2.0f), d2, d1);  // 3 d_2 - t_1
  const float2 e2 = __ffma2_rn(f2(-0.5f), t2, __fmul2_rn(f2(1.5f), d2));
  const float2 num = __ffma2_rn(p0, e0, __ffma2_rn(p1, e1, __fmul2_rn(p2, e2)));
  const float2 den = __ffma2_rn(f2(6.0f), p1, __ffma2_rn(f2(3.0f), p2, p0));
  return __ffma2_rn(num, rcp2(den), v2);
}

}  // namespace mth
