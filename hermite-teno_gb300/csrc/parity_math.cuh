// Bit-reproducible FP64 numerics of the plain path.
//
// Why: TENO's cut-off is a discontinuous decision.  In the tails of waves the data vary by
// ~1e-10 relative to their magnitude, so a rounding difference in the characteristic values
// (1e-16 absolute) can move a weight across the cut-off; the flip then changes the solution by
// ~1e-10.  Agreement with the reference to 1e-12 over hundreds of steps therefore needs the same
// rounding, not just the same formulas.  Every function here performs exactly the IEEE
// operations, in exactly the order, of the reference's expressions (reductions left to right),
// and this header is only compiled in translation units built with --fmad=false so that no
// multiply-add is fused.  Divisions and square roots are IEEE correctly rounded, as on the CPU.
//
// The one deliberate difference: the TENO cut-off weights (1 + tau/(SI+eps))^6 / sum only select
// one of 8 cut-off patterns, so they are compared in float (the ratios of the weights' bases to
// the largest, from SI + eps and tau scaled into float range, and their sixth powers); when a
// weight lies within a guard band of the threshold (several times the float evaluation's error
// bound), the decision is recomputed with the reference's divisions and pow.  The indicators and
// tau themselves are the reference's bits.  The reconstructed values use the pattern's weights
// from a table built with the reference's own normalisation, so they are bit-identical.
#pragma once

#include "device_math.cuh"
#include "fp3.cuh"
#include "mixed_conv.cuh"
#include "hermite_math.cuh"

namespace hteno {
namespace par {

// Tests on a double's bits, on the integer pipes: the FP64 pipe (1/64 of the FP32 rate on GB300)
// is left to the arithmetic.  Exactly the IEEE predicates: x == 0.0 (either sign), isnan(x).
__device__ __forceinline__ bool zero_bits(double x) {
  return (static_cast<unsigned long long>(__double_as_longlong(x)) << 1) == 0ull;
}
__device__ __forceinline__ bool nan_bits(double x) {
  return (static_cast<unsigned long long>(__double_as_longlong(x)) & 0x7fffffffffffffffull) >
         0x7ff0000000000000ull;
}
__device__ __forceinline__ double catchnan(double x) { return nan_bits(x) ? 1e-15 : x; }

// dot of a 3-vector of coefficients with u[0..2], left to right (Eigen .dot in the reference)
__device__ __forceinline__ fp dot3(fp c0, fp c1, fp c2, const fp* u) {
  fp s = c0 * u[0];
  s = s + c1 * u[1];
  s = s + c2 * u[2];
  return s;
}
__device__ __forceinline__ fp dot3v(const fp* p, const fp* w) {
  fp s = p[0] * w[0];
  s = s + p[1] * w[1];
  s = s + p[2] * w[2];
  return s;
}
// column k of a coefficient table in global memory . u
template <int N>
__device__ __forceinline__ fp dot3t(const double (&t)[3][N], int k, const fp* u) {
  return dot3(ldk(t[0][k]), ldk(t[1][k]), ldk(t[2][k]), u);
}
// p . the three weights at w (global memory)
__device__ __forceinline__ fp dot3w(const fp* p, const double* w) {
  const fp ww[3] = {ldk(w[0]), ldk(w[1]), ldk(w[2])};
  return dot3v(p, ww);
}

// Correctly rounded a / b for several numerators over one denominator: y = RN(1/b) once, then per
// numerator q0 = RN(a y), r = a - b q0 (exact, one FMA), q = RN(q0 + r y).  By Markstein's theorem
// (Markstein, IBM J. Res. Dev. 34(1), 1990; Muller et al., Handbook of Floating-Point Arithmetic,
// 2018, Sec. 4.7) q is a / b correctly rounded when y is within half an ulp of 1/b and q0 within
// one ulp of a / b, barring underflow and overflow: 3 FP64 operations per quotient instead of a
// division's ~10.  Operands outside [2^-500, 2^501) in magnitude (subnormals, infinities, NaN) take
// the division itself, so the theorem's conditions hold wherever the short form is used; a
// numerator of +0 gives q0 = r = q = 0 with the division's sign, so it takes the short form too.
struct Den {
  fp b, y;
  bool ok;
};
__device__ __forceinline__ bool mid_range(double x) {
  const unsigned e = (unsigned(__double2hiint(x)) >> 20) & 0x7ffu;
  return e - 523u <= 1000u;  // biased exponent in [523, 1523]
}
__device__ __forceinline__ Den den_of(fp b) { return Den{b, __drcp_rn(b.v), mid_range(b.v)}; }
// a denominator known at compile time, from its value and RN(1 / value) in the table
__device__ __forceinline__ Den den_lit(double b, Lit y) { return Den{b, lit(y), true}; }
// Not inlined: hardly ever taken, and a division's code at each quotient crowds the instruction cache
// (FV 2D FP64 1024^2, two steps: 48.5 -> 47.8 ms; 64 x 48: 13.9 -> 13.1).
static __device__ __noinline__ double divide(double a, double b) { return a / b; }
__device__ __forceinline__ fp quot(fp a, const Den& d) {
  if (d.ok && (mid_range(a.v) || __double_as_longlong(a.v) == 0ll)) {
    const fp q0 = a * d.y;
    const double r = fma(-d.b.v, q0.v, a.v);
    return fma(r, d.y.v, q0.v);
  }
  return divide(a.v, d.b.v);
}

// a / c correctly rounded for the integers c whose 1/c is in the table as hi + lo (kDivC, kDivCLo: 1/c
// rounded, and what that leaves, rounded): RN(a hi + RN(a lo)), two operations.  (Multiplication by a
// constant in two parts, Brisebarre & Muller, IEEE Trans. Computers 57(2), 2008.)  The value that is
// rounded is off by less than 2^-104 of itself, 2^-51 ulp, while a / c, a quotient by an integer with
// the odd part d, lies 1/(2d) ulp or more from every midpoint of two doubles (d <= 315 here): no
// rounding can differ.  +0 stays +0, and -0 keeps its sign where the low part is positive; where it is
// negative (6720, 1680) -0 would give +0: callers pass absolute values there.  Other operands outside quot's
// range take the division.
__device__ __forceinline__ fp quot_lit(fp a, double c, Lit hi) {
  if (mid_range(a.v) || zero_bits(a.v)) return fma(a.v, lit(hi).v, (a * lit(Lit(hi + 1))).v);
  return divide(a.v, c);
}

// q0 + 2 x where 2 x overflows by itself, whatever q0 is
static __device__ __noinline__ double plus_twice_huge(double x, double q0) { return __dadd_rn(q0, __dmul_rn(2.0, x)); }

// Schemes::SSPRK::RungeKuttaIII (Schemes_SSPRK.cpp:3-15)
__device__ __forceinline__ double rk3(fp q0, fp qn, fp rhs, fp dt, int stage) {
  if (stage == 1) return (q0 + dt * rhs).v;
  const fp x = qn + rhs * dt;
  // (the quarter rounds where it is subnormal: not folded into the sum)
  if (stage == 2) return (lit(kThreeQuarters) * q0 + lit(kQuarter) * x).v;
  fp s = scaled(kTwo, x, q0);
  if (__builtin_expect((unsigned(__double2hiint(x.v)) & 0x7ff00000u) == 0x7fe00000u, 0)) s = plus_twice_huge(x.v, q0.v);
  return quot_lit(s, 3.0, kDiv3).v;
}
// x <= 0, on the integer pipes
__device__ __forceinline__ bool nonpositive_bits(double x) {
  return __double_as_longlong(x) <= 0ll && !nan_bits(x);
}

// ---- Schemes::Lagrange ----------------------------------------------------------------------

// smoothnessMeasure (Schemes_Lagrange.cpp:1013-1026).  The b are halved term by term (exact
// scalings by powers of two of the reference's b / 2).
__device__ __forceinline__ void lagrange_si(const fp* v, fp* SI) {
  fp c[3], b[3];
  const fp m2 = lit(kThreeHalves) * v[2];
  c[0] = scaled(kNegTwo, v[3], v[2]) + v[4];
  b[0] = scaled(kHalf, v[4], scaled(kNegTwo, v[3], m2));
  c[1] = scaled(kNegTwo, v[2], v[1]) + v[3];
  b[1] = scaled(kNegHalf, v[3], lit(kHalf) * v[1]);
  c[2] = scaled(kNegTwo, v[1], v[0]) + v[2];
  b[2] = scaled(kNegTwo, v[1], lit(kHalf) * v[0]) + m2;
#pragma unroll
  for (int k = 0; k < 3; ++k) SI[k] = b[k] * b[k] + lit(kThirteenTwelfths) * c[k] * c[k];
}
// fullpointsSmootness (:1029-1034)
__device__ __forceinline__ fp lagrange_b35(const fp* v) {
  const fp r = v[4] * (lit(k6908) * v[4] - lit(k51001) * v[3] + lit(k67923) * v[2] - lit(k38947) * v[1] +
                       lit(k8209) * v[0]) +
               v[3] * (lit(k104963) * v[3] - lit(k299076) * v[2] + lit(k179098) * v[1] - lit(k38947) * v[0]) +
               v[2] * (lit(k231153) * v[2] - lit(k299076) * v[1] + lit(k67923) * v[0]) +
               v[1] * (lit(k104963) * v[1] - lit(k51001) * v[0]) + lit(k6908) * v[0] * v[0];
  return quot_lit(r, 5040.0, kDiv5040);
}

// 1/x to a relative 2^-45 for the cut-off decision only (never for a value that is kept): a
// float reciprocal of x's significand (rcp.approx.ftz.f32, on the MUFU pipe), rescaled by x's
// exponent on the integer pipes, and one Newton step in double (2 FMAs instead of the ~10 FP64
// operations of a correctly rounded reciprocal).  Exponents near the ends of the range, zeros,
// infinities and NaN take the correctly rounded reciprocal.
__device__ __forceinline__ double decision_rcp(double x) {
  const unsigned hx = unsigned(__double2hiint(x)), lx = unsigned(__double2loint(x));
  const unsigned ex = (hx >> 20) & 0x7ffu;
  if (ex - 64u > 1916u) return __drcp_rn(x);
  const float m = __uint_as_float(0x3f800000u | ((hx & 0xfffffu) << 3) | (lx >> 29));
  float rf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(m));
  const unsigned r = __float_as_uint(rf), er = (r >> 23) & 0xffu, mr = r & 0x7fffffu;
  const unsigned hy = (hx & 0x80000000u) | ((er + 2046u - 127u - ex) << 20) | (mr >> 3);
  const double y = __hiloint2double(int(hy), int(mr << 29));
  return fma(y, fma(-x, y, 1.0), y);
}

// Largest r whose sixth power is finite with margin (pow(2e51, 6) = 6.4e306): beyond it the
// reference's weights overflow to inf and its normalised weights are NaN.
constexpr double kPow6Max = 2e51;

// The fast part of a cut-off decision, in float, from the ratios x_k = r_k / r_max (in (0, 1],
// or NaN): a_k = x_k^6, kept where a_k >= ct * (a_0 + a_1 + a_2).  Any a_k farther than `band` of
// the limit from it is decided as exact arithmetic decides it (the callers' error bounds are a
// fraction of the band); nearer ones set *near and the caller takes the reference's own
// arithmetic.  NaN ratios compare false, as in double.  (The FP64 pipe runs at 1/64 of the float
// rate on GB300.)
__device__ __forceinline__ int cutoff_core(const float* x, float ct, float band, bool* near) {
  float a[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float x2 = x[k] * x[k];
    a[k] = (x2 * x2) * x2;
  }
  const float lim = ct * ((a[0] + a[1]) + a[2]);
  int pat = 0;
  bool nr = false;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    pat |= (a[k] < lim ? 0 : 1) << k;
    nr |= fabsf(a[k] - lim) <= band * lim;
  }
  *near = nr;
  return pat;
}
// ... from double ratios (converted on the integer pipes): the float chain's relative error is
// below 1e-6 (x_k to 2^-24, six roundings in a_k, two in the sum), well inside a band of 1e-5.
__device__ __forceinline__ int cutoff_fast(const double* x, double ct, bool* near) {
  const float xf[3] = {mix::d2f(x[0]), mix::d2f(x[1]), mix::d2f(x[2])};
  return cutoff_core(xf, float(ct), 1e-5f, near);
}

// The ratios x_k = r_k / r_max of r_k = 1 + tau / d_k in float, without reciprocals or r_k's
// range: with d_min = min d_k, x_k = (d_min / d_k) (d_k + tau) / (d_min + tau).  The four doubles
// are first scaled by one power of two (exponent bits, on the integer pipes) so that the largest
// lies in [1, 2).  Relative error of x_k below 2^-19.7 (four inputs rounded to float, two
// __fdividef quotients of 2 ulp and three roundings), so of a_k below 7.4e-6.  False when a value
// is NaN, infinite, subnormal or more than 2^125 below the largest (the caller takes the double
// path).  d_k > 0 and tau >= 0 here; within 2^125 every r_k <= 1 + 2^126 < kPow6Max, so the
// reference's weights are finite.
__device__ __forceinline__ bool scaled_ratios(const double* d, double tau, float* x) {
  const double v[4] = {d[0], d[1], d[2], tau};
  int hi[4];
  unsigned lo[4], e[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    hi[i] = __double2hiint(v[i]);
    lo[i] = unsigned(__double2loint(v[i]));
    e[i] = (unsigned(hi[i]) >> 20) & 0x7ffu;
  }
  const unsigned em = max(max(e[0], e[1]), max(e[2], e[3]));
  // (the callers' indicators are sums of squares and tau an absolute value or a maximum of them;
  // a sign bit, even of -0, sends the decision to the double path all the same)
  if (em == 0x7ffu || (hi[0] | hi[1] | hi[2] | hi[3]) < 0) return false;
  float f[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (i == 3 && ((unsigned(hi[3]) << 1) | lo[3]) == 0u) {
      f[3] = 0.0f;  // tau = 0: every r_k is 1
    } else {
      if (e[i] == 0u || e[i] + 125u < em) return false;
      // scaled exponent e - em + 1023 in [898, 1023]: a normal float in [2^-125, 2)
      f[i] = mix::d2f(__hiloint2double(hi[i] - (int(em) - 1023) * (1 << 20), int(lo[i])));
    }
  }
  const float dmin = fminf(fminf(f[0], f[1]), f[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k)
    x[k] = __fdividef(dmin, f[k]) * __fdividef(f[k] + f[3], dmin + f[3]);
  return true;
}

// Cut-off pattern of the reference's cutOff() (:1141-1149) given SI and tau.  Fast path: the
// ratios in float from d_k = SI_k + epsz and tau (scaled_ratios, guard band 2^-13 relative, eight
// times its error bound), or in double where the scaling cannot reach (guard band 1e-5); inside
// the band the reference's arithmetic decides.
__device__ __forceinline__ int cutoff_pattern(const fp* SI, double tau, double ct) {
  constexpr double epsz = HTENO_LAG_EPSZ;  // of the Hermite schemes too
  const double d[3] = {(SI[0] + lit(kEpsz)).v, (SI[1] + lit(kEpsz)).v, (SI[2] + lit(kEpsz)).v};
  float xf[3];
  bool near;
  int pat;
  if (scaled_ratios(d, tau, xf)) {
    pat = cutoff_core(xf, float(ct), 0x1p-13f, &near);
  } else {
    double r[3], x[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = 1.0 + tau * decision_rcp(d[k]);
    const double rm = fmax(fmax(r[0], r[1]), r[2]);
    const double inv = decision_rcp(rm);
#pragma unroll
    for (int k = 0; k < 3; ++k) x[k] = r[k] * inv;
    pat = cutoff_fast(x, ct, &near);
    // where pow(r, 6) overflows the reference's weights are inf / inf = NaN (a kept candidate):
    // its own arithmetic decides
    near = near || !(rm < kPow6Max);
  }
  if (near) {  // reference arithmetic: w_k = pow(1 + tau/(SI_k + epsz), 6) / sum
    double w[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) w[k] = pow(1.0 + tau / (SI[k].v + epsz), 6.0);
    const double s = (w[0] + w[1]) + w[2];
    pat = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) pat |= ((w[k] / s) < ct ? 0 : 1) << k;
  }
  return pat;
}

// The cut-off pattern of one side of teno5 (:481-511) / teno5i (:1235-1263) for the window v with
// indicators SI (bit k set: candidate k kept).
__device__ __forceinline__ int teno_decide(const fp* v, const fp* SI, bool improved) {
  // All three indicators exactly zero (constant data): the three ratios 1 + tau/(0 + epsz) are
  // equal whatever tau is, and the cut-off keeps all candidates (pattern 7) -- decided without
  // tau, same bits.  (Equal values alone do not suffice: 3u - 4u + u can leave a rounding
  // residue in one indicator.)
  // The full arithmetic below gives pattern 7 on such a window too (three equal ratios): a thread that
  // returns here only saves it.
  if (zero_bits(SI[0].v) && zero_bits(SI[1].v) && zero_bits(SI[2].v)) return 7;
  double tau;
  if (!improved) {
    const fp b35 = lagrange_b35(v);
    const fp mean = quot_lit(scaled(kFour, SI[1], SI[0] + SI[2]), 6.0, kDiv6);
    tau = fabs((b35 - mean).v);
  } else {
    tau = SI[0].v;
    tau = (tau < SI[1].v) ? SI[1].v : tau;
    tau = (tau < SI[2].v) ? SI[2].v : tau;
  }
  return cutoff_pattern(SI, tau, HTENO_LAG_CT);
}

// One side of teno5 / teno5i given the candidates p and stencil v.
__device__ __forceinline__ double teno_side_si(const DevConst& C, const fp* p, const fp* v,
                                               const fp* SI, int side, bool improved) {
  const int pat = teno_decide(v, SI, improved);
  return catchnan(dot3w(p, side ? C.wtab_p[pat] : C.wtab_m[pat]).v);
}
__device__ __forceinline__ double teno_side(const DevConst& C, const fp* p, const fp* v,
                                            int side, bool improved) {
  fp SI[3];
  lagrange_si(v, SI);
  return teno_side_si(C, p, v, SI, side, improved);
}

// ---- the selectable alternatives (Schemes_Lagrange.cpp:358-594, 1265-1294), one side each ----

// Cut-off pattern from the exact ratios r_k, whose sixth powers are the reference's raw weights:
// fast path on (r_k / r_max)^6 with a guard band, the reference's pow-and-divide inside it.
__device__ __forceinline__ int cutoff_from_r(const double* r, double ct) {
  const double rm = fmax(fmax(r[0], r[1]), r[2]);
  const double inv = __drcp_rn(rm);
  double x[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) x[k] = r[k] * inv;
  bool near;
  int pat = cutoff_fast(x, ct, &near);
  if (near || !(rm < kPow6Max)) {  // the reference's arithmetic (also where pow(r, 6) overflows)
    double w[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) w[k] = pow(r[k], 6.0);
    const double s = (w[0] + w[1]) + w[2];
    pat = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) pat |= ((w[k] / s) < ct ? 0 : 1) << k;
  }
  return pat;
}

__device__ __forceinline__ double normalised(const double* p, double* w) {
  const double s = (w[0] + w[1]) + w[2];
#pragma unroll
  for (int k = 0; k < 3; ++k) w[k] = w[k] / s;
  double o = p[0] * w[0];
  o = o + p[1] * w[1];
  o = o + p[2] * w[2];
  return catchnan(o);
}

// weno5N / teno5N indicators (:445-450) on the side's window v[0..4]; returns the 5-point
// difference |v0 - 4v1 + 6v2 - 4v3 + v4|
__device__ __forceinline__ double n_indicators(const double* v, double* SI) {
  SI[2] = 0.1 * fabs(v[0] - 3.0 * v[1] + 2.0 * v[2]) + fabs(v[0] - 2.0 * v[1] + v[2]);
  SI[1] = 0.1 * fabs(v[3] - v[2]) + fabs(v[1] - 2.0 * v[2] + v[3]);
  SI[0] = 0.1 * fabs(v[3] - v[2]) + fabs(v[2] - 2.0 * v[3] + v[4]);
  return fabs(v[0] - 4.0 * v[1] + 6.0 * v[2] - 4.0 * v[3] + v[4]);
}

// kind 3 weno5JS, 4 weno5Z, 5 weno5N, 6 teno5N, 7 teno5a
__device__ __forceinline__ double alt_side(const DevConst& C, int kind, const double* p,
                                           const double* v, int side) {
  const double* d = side ? C.dkp : C.dkm;
  double SI[3], w[3];
  if (kind == 3 || kind == 4 || kind == 7) {
    const fp vf[5] = {v[0], v[1], v[2], v[3], v[4]};
    fp S[3];
    lagrange_si(vf, S);
#pragma unroll
    for (int k = 0; k < 3; ++k) SI[k] = S[k].v;
  }
  if (kind == 3) {  // w_k = d_k / (eps + SI_k)^2
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double e = HTENO_LAG_EPS + SI[k];
      w[k] = d[k] / (e * e);
    }
    return normalised(p, w);
  }
  if (kind == 4) {  // tau = |SI_2 - SI_0|, w_k = d_k (1 + tau / (SI_k + epsz))
    const double tau = fabs(SI[2] - SI[0]);
#pragma unroll
    for (int k = 0; k < 3; ++k) w[k] = d[k] * (1.0 + (tau / (SI[k] + HTENO_LAG_EPSZ)));
    return normalised(p, w);
  }
  if (kind == 5) {  // tau = |5-point difference|^2.5, w_k = d_k (1 + tau / (SI_k + eps)^2)
    const double tau = pow(n_indicators(v, SI), 2.5);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double e = SI[k] + HTENO_LAG_EPS;
      w[k] = d[k] * (1.0 + (tau / (e * e)));
    }
    return normalised(p, w);
  }
  double r[3];
  if (kind == 6) {  // r_k = 1 + tau / (SI_k + eps)^2, tau = |5-point difference|^2
    const double x = n_indicators(v, SI);
    const double tau = x * x;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const double e = SI[k] + HTENO_LAG_EPS;
      r[k] = 1.0 + tau / (e * e);
    }
  } else {  // teno5a: r_k = 1 / (SI_k + epsz)
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = 1.0 / (SI[k] + HTENO_LAG_EPSZ);
  }
  const int pat = cutoff_from_r(r, HTENO_LAG_CT);
  const fp pf[3] = {p[0], p[1], p[2]};
  return catchnan(dot3w(pf, side ? C.wtab_p[pat] : C.wtab_m[pat]).v);
}

// kind 2 linear (:1219-1233) or an alternative (3..7), one side, from its candidates and window
__device__ __forceinline__ double other_side(const DevConst& C, int kind, const fp* p, const fp* v, int side) {
  if (kind == 2) return dot3w(p, side ? C.dkp : C.dkm).v;
  const double pd[3] = {p[0].v, p[1].v, p[2].v};
  const double vd[5] = {v[0].v, v[1].v, v[2].v, v[3].v, v[4].v};
  return alt_side(C, kind, pd, vd, side);
}

// kind 0 teno5, 1 teno5i, 2 linear (:1219-1233), 3..7 the alternatives above.  C in global memory.
__device__ __forceinline__ void lagrange_recon(const DevConst& C, int kind, const double* ud,
                                               double& outm, double& outp) {
  const fp u[6] = {ud[0], ud[1], ud[2], ud[3], ud[4], ud[5]};
  fp p[3], pp[3];
  p[0] = dot3t(C.crj, 1, u + 2);
  p[1] = dot3t(C.crj, 2, u + 1);
  p[2] = dot3t(C.crj, 3, u + 0);
  // the two sides' windows overlap in 5 cells: p1+ = p0-, p2+ = p1- (the same expressions on the
  // same operands, the same bits)
  pp[0] = dot3t(C.crj, 0, u + 3);
  pp[1] = p[0];
  pp[2] = p[1];
  if (kind <= 1) {
    // teno5 / teno5i: two of the indicators' second-difference terms are shared as well
    fp c[4], t[4], SIm[3], SIp[3], bm[3], bp[3];
    c[0] = scaled(kNegTwo, u[3], u[2]) + u[4];
    c[1] = scaled(kNegTwo, u[2], u[1]) + u[3];
    c[2] = scaled(kNegTwo, u[1], u[0]) + u[2];
    c[3] = scaled(kNegTwo, u[4], u[3]) + u[5];  // c0 of the + side
#pragma unroll
    for (int k = 0; k < 4; ++k) t[k] = lit(kThirteenTwelfths) * c[k] * c[k];
    const fp m2 = lit(kThreeHalves) * u[2], m3 = lit(kThreeHalves) * u[3];
    const fp h1 = lit(kHalf) * u[1];
    bm[0] = scaled(kHalf, u[4], scaled(kNegTwo, u[3], m2));
    bm[1] = scaled(kNegHalf, u[3], h1);
    bm[2] = scaled(kNegTwo, u[1], lit(kHalf) * u[0]) + m2;
    bp[0] = scaled(kHalf, u[5], scaled(kNegTwo, u[4], m3));
    bp[1] = scaled(kNegHalf, u[4], lit(kHalf) * u[2]);
    bp[2] = scaled(kNegTwo, u[2], h1) + m3;
    SIm[0] = bm[0] * bm[0] + t[0];
    SIm[1] = bm[1] * bm[1] + t[1];
    SIm[2] = bm[2] * bm[2] + t[2];
    SIp[0] = bp[0] * bp[0] + t[3];
    SIp[1] = bp[1] * bp[1] + t[0];
    SIp[2] = bp[2] * bp[2] + t[1];
    outm = teno_side_si(C, p, u, SIm, 0, kind == 1);
    outp = teno_side_si(C, pp, u + 1, SIp, 1, kind == 1);
    return;
  }
  outm = other_side(C, kind, p, u, 0);
  outp = other_side(C, kind, pp, u + 1, 1);
}

// lagrange_recon out of line, the stencil by value: the face kernels reconstruct four fields, and four
// inlined copies overflow the instruction cache.
struct SidePair {
  double m, p;
};
static __device__ __noinline__ SidePair recon_call(const DevConst& C, int kind, double u0, double u1, double u2,
                                                   double u3, double u4, double u5) {
  const double u[6] = {u0, u1, u2, u3, u4, u5};
  SidePair o;
  lagrange_recon(C, kind, u, o.m, o.p);
  return o;
}

// One side of lagrange_recon (side 0: u^-, side 1: u^+), the same arithmetic.
__device__ __forceinline__ double lagrange_side(const DevConst& C, int kind, const double* ud, int side) {
  const fp v[5] = {side ? ud[1] : ud[0], side ? ud[2] : ud[1], side ? ud[3] : ud[2], side ? ud[4] : ud[3],
                   side ? ud[5] : ud[4]};
  // candidate k is column 1 + k - side of crj on the cells from 2 - k of the window
  fp p[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) p[k] = dot3t(C.crj, 1 + k - side, v + 2 - k);
  return kind <= 1 ? teno_side(C, p, v, side, kind == 1) : other_side(C, kind, p, v, side);
}


// weno5JS3PointsQuadrature (Schemes_Lagrange.cpp:1155-1217).  Not inlined: the flux kernels call
// it 8 times per face, and eight inlined copies overflow the instruction cache.  C in global memory.
static __device__ __noinline__ void gl3(const DevConst& C, const double* ud, double* out) {
  const fp u[5] = {ud[0], ud[1], ud[2], ud[3], ud[4]};
  fp bg[3], cg[3], s2[3];
  const fp m2 = lit(kThree) * u[2];
  bg[0] = scaled(kNegFour, u[1], u[0]) + m2;
  cg[0] = scaled(kNegTwo, u[1], u[0]) + u[2];
  bg[1] = u[1] - u[3];
  cg[1] = scaled(kNegTwo, u[2], u[1]) + u[3];
  bg[2] = scaled(kNegFour, u[3], m2) + u[4];
  cg[2] = scaled(kNegTwo, u[3], u[2]) + u[4];
  const fp n2 = lit(k23) * u[2];
  fp p[3];
  // (taken only when every active lane of the warp can take it: the full arithmetic gives the same
  // bits on constant data, and a warp then never runs both)
  if (__all_sync(__activemask(), zero_bits(bg[0].v) && zero_bits(bg[1].v) && zero_bits(bg[2].v) &&
                                     zero_bits(cg[0].v) && zero_bits(cg[1].v) && zero_bits(cg[2].v))) {
    // every indicator is zero: the normalised weights are the constants gl3flat, which the host
    // computed with these same operations -- the same bits without the 24 divisions
#pragma unroll
    for (int k = 0; k < 3; ++k) p[k] = dot3t(C.gp, k, u + k);
    out[0] = dot3w(p, C.gl3flat[0]).v;
    p[0] = quot_lit(scaled(kTwo, u[1], -u[0]) + n2, 24.0, kDiv24);
    p[1] = quot_lit(-u[1] + lit(k26) * u[2] - u[3], 24.0, kDiv24);
    p[2] = quot_lit(scaled(kTwo, u[3], n2) - u[4], 24.0, kDiv24);
    fp c = fp(ldk(C.sumw0p)) * dot3w(p, C.gl3flat[1]);
    c = c - fp(ldk(C.sumw0m)) * dot3w(p, C.gl3flat[2]);
    out[1] = c.v;
#pragma unroll
    for (int k = 0; k < 3; ++k) p[k] = dot3t(C.gm, k, u + k);
    out[2] = dot3w(p, C.gl3flat[3]).v;
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k] = catchnan(out[k]);
    return;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    // 0.25 bg^2 + 13/12 cg^2, the first product exact
    const fp si = scaled(kQuarter, bg[k] * bg[k], lit(kThirteenTwelfths) * (cg[k] * cg[k]));
    const fp e = lit(kEps6) + si;
    s2[k] = e * e;  // pow(eps + SI, 2)
  }
  const Den ds[3] = {den_of(s2[0]), den_of(s2[1]), den_of(s2[2])};  // each serves 4 weight sets
  auto weighted = [&](const double* lw) {
    fp w[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) w[k] = quot(ldk(lw[k]), ds[k]);
    const Den dn = den_of((w[0] + w[1]) + w[2]);
#pragma unroll
    for (int k = 0; k < 3; ++k) w[k] = quot(w[k], dn);
    return dot3v(p, w);
  };
#pragma unroll
  for (int k = 0; k < 3; ++k) p[k] = dot3t(C.gp, k, u + k);
  out[0] = weighted(C.linwp).v;
  p[0] = quot_lit(scaled(kTwo, u[1], -u[0]) + n2, 24.0, kDiv24);
  p[1] = quot_lit(-u[1] + lit(k26) * u[2] - u[3], 24.0, kDiv24);
  p[2] = quot_lit(scaled(kTwo, u[3], n2) - u[4], 24.0, kDiv24);
  fp c = fp(ldk(C.sumw0p)) * weighted(C.linw0p);
  c = c - fp(ldk(C.sumw0m)) * weighted(C.linw0m);
  out[1] = c.v;
#pragma unroll
  for (int k = 0; k < 3; ++k) p[k] = dot3t(C.gm, k, u + k);
  out[2] = weighted(C.linwm).v;
#pragma unroll
  for (int k = 0; k < 3; ++k) out[k] = catchnan(out[k]);
}

// ---- Equations::Euler2D ---------------------------------------------------------------------

// y - x / 2, the energy less the kinetic part, in one operation.  Where the half may be subnormal the reference
// rounds it first.  That can reach the result only if y is below 2^-968 (the half is below 2^-1021 there):
// such y take the separate operations.  The test needs y alone, on the integer pipes beside the chain.
__device__ __forceinline__ bool tiny(fp y) { return (unsigned(__double2hiint(y.v)) & 0x7fffffffu) < (123u << 20); }  // 2^-900
static __device__ __noinline__ double minus_half_tiny(double x, double y) { return __dsub_rn(y, __dmul_rn(0.5, x)); }
__device__ __forceinline__ fp minus_half(fp x, fp y) {
  if (__builtin_expect(tiny(y), 0)) return minus_half_tiny(x.v, y.v);
  return scaled(kNegHalf, x, y);
}
__device__ __forceinline__ fp operator/(fp a, fp b) { return fp(a.v / b.v); }
__device__ __forceinline__ fp sqrt_abs(fp a) { return fp(sqrt(fabs(a.v))); }
__device__ __forceinline__ fp max_(fp a, fp b) { return fp(fmax(a.v, b.v)); }

// The divisions by a density share one correctly rounded reciprocal: d = den_of(q[0]).
__device__ __forceinline__ void primitive(double g1, const fp* q, const Den& d, fp* w) {  // :20-26
  w[0] = q[0];
  w[1] = quot(q[1], d);
  w[2] = quot(q[2], d);
  w[3] = minus_half(q[1] * w[1] + q[2] * w[2], q[3]) * g1;
}
__device__ __forceinline__ void primitive(double g1, const double* q, double* w) {
  const fp qf[4] = {q[0], q[1], q[2], q[3]};
  fp wf[4];
  primitive(g1, qf, den_of(qf[0]), wf);
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = wf[k].v;
}

__device__ __forceinline__ void flux(int dir, const fp* q, const fp* w, fp* f) {
  if (dir == 1) {
    f[0] = q[1];
    f[1] = q[1] * w[1] + w[3];
    f[2] = q[1] * w[2];
    f[3] = w[1] * (q[3] + w[3]);
  } else {
    f[0] = q[2];
    f[1] = q[2] * w[1];
    f[2] = q[2] * w[2] + w[3];
    f[3] = w[2] * (q[3] + w[3]);
  }
}

// Face eigensystem (eigen2DEuler, FV_System2D.cpp:265-361): the entries of R and L are kept as
// the scalars the reference's matrices are built from.
struct Eig {
  fp vxm, vym, hm, qm, cm, t0r;  // t0r = vn * cm (right eigenvectors)
  fp rcm, b1, b2, s0, s1, t2;    // left eigenvectors
};

__device__ __forceinline__ Eig eig(double g1, int dir, fp sra, fp ua, fp va, fp ha, fp srb, fp ub,
                                   fp vb, fp hb) {
  Eig e;
  const fp t0 = sra / (sra + srb);
  const fp t1 = lit(kOne) - t0;
  e.vxm = t0 * ua + t1 * ub;
  e.vym = t0 * va + t1 * vb;
  e.hm = t0 * ha + t1 * hb;
  e.qm = lit(kHalf) * (e.vxm * e.vxm + e.vym * e.vym);
  e.cm = sqrt_abs(fp(g1) * (e.hm - e.qm));
  const fp vn = dir == 1 ? e.vxm : e.vym;
  e.t0r = vn * e.cm;
  e.rcm = lit(kOne) / e.cm;
  e.b1 = fp(g1) * e.rcm * e.rcm;
  e.b2 = e.qm * e.b1;
  e.s0 = vn * e.rcm;
  e.s1 = e.b1 * vn;
  e.t2 = lit(kHalf) * e.b1;
  return e;
}

// The eigensystem from its seven stored scalars (vxm, vym, hm, qm, cm, rcm, b1 with `stride`
// between them), the derived ones recomputed with the same operations.
__device__ __forceinline__ Eig eig_load(int dir, const double* f, size_t stride) {
  Eig e;
  e.vxm = f[0];
  e.vym = f[stride];
  e.hm = f[2 * stride];
  e.qm = f[3 * stride];
  e.cm = f[4 * stride];
  e.rcm = f[5 * stride];
  e.b1 = f[6 * stride];
  const fp vn = dir == 1 ? e.vxm : e.vym;
  e.t0r = vn * e.cm;
  e.b2 = e.qm * e.b1;
  e.s0 = vn * e.rcm;
  e.s1 = e.b1 * vn;
  e.t2 = lit(kHalf) * e.b1;
  return e;
}
__device__ __forceinline__ void eig_store(const Eig& e, double* f, size_t stride) {
  f[0] = e.vxm.v;
  f[stride] = e.vym.v;
  f[2 * stride] = e.hm.v;
  f[3 * stride] = e.qm.v;
  f[4 * stride] = e.cm.v;
  f[5 * stride] = e.rcm.v;
  f[6 * stride] = e.b1.v;
}

// L * q with the reference's left-to-right row sums (leftEigenVectorx/y, :133-205).  Zero entries
// of L add exact zeros in the reference and are skipped; unit entries multiply exactly.
__device__ __forceinline__ void left(const Eig& e, int dir, const fp* q, fp* c) {
  const fp half = lit(kHalf), nhalf = lit(kNegHalf);
  const fp l00 = half * (e.b2 + e.s0), l0n = nhalf * (e.s1 + e.rcm);
  const fp l30 = half * (e.b2 - e.s0), l3n = nhalf * (e.s1 - e.rcm);
  const fp l20 = lit(kOne) - e.b2;
  if (dir == 1) {
    const fp lt = -e.t2 * e.vym, l2t = e.b1 * e.vym;
    fp s = l00 * q[0]; s = s + l0n * q[1]; s = s + lt * q[2]; s = s + e.t2 * q[3]; c[0] = s;
    s = -e.vym * q[0]; s = s + q[2]; c[1] = s;
    s = l20 * q[0]; s = s + e.s1 * q[1]; s = s + l2t * q[2]; s = s + (-e.b1) * q[3]; c[2] = s;
    s = l30 * q[0]; s = s + l3n * q[1]; s = s + lt * q[2]; s = s + e.t2 * q[3]; c[3] = s;
  } else {
    const fp lt = -e.t2 * e.vxm, l2t = e.b1 * e.vxm;
    fp s = l00 * q[0]; s = s + lt * q[1]; s = s + l0n * q[2]; s = s + e.t2 * q[3]; c[0] = s;
    s = -e.vxm * q[0]; s = s + q[1]; c[1] = s;
    s = l20 * q[0]; s = s + l2t * q[1]; s = s + e.s1 * q[2]; s = s + (-e.b1) * q[3]; c[2] = s;
    s = l30 * q[0]; s = s + lt * q[1]; s = s + l3n * q[2]; s = s + e.t2 * q[3]; c[3] = s;
  }
}
// Row r of left() by itself, its four entries in the order of q; row 1 is (-v_t, 0, 1, 0) with the
// unit at the tangential momentum.
struct LeftRow {
  fp a[4];
  bool unit, dirx;
  __device__ __forceinline__ fp dot(fp q0, fp q1, fp q2, fp q3) const {
    fp s = a[0] * q0;
    if (unit) return s + (dirx ? q2 : q1);
    s = s + a[1] * q1;
    s = s + a[2] * q2;
    return s + a[3] * q3;
  }
};
__device__ __forceinline__ LeftRow left_row(const Eig& e, int dir, int r) {
  const fp vt = dir == 1 ? e.vym : e.vxm;
  const bool r0 = r == 0, r2 = r == 2;
  // rows 0 and 3 differ in the sign of s0 and rcm
  const fp s0 = r0 ? e.s0 : -e.s0, rcm = r0 ? e.rcm : -e.rcm;
  const fp c0 = r2 ? lit(kOne) - e.b2 : lit(kHalf) * (e.b2 + s0);
  const fp cn = r2 ? e.s1 : lit(kNegHalf) * (e.s1 + rcm);
  const fp ct = (r2 ? e.b1 : -e.t2) * vt;
  LeftRow L;
  L.a[0] = r == 1 ? -vt : c0;
  L.a[1] = dir == 1 ? cn : ct;
  L.a[2] = dir == 1 ? ct : cn;
  L.a[3] = r2 ? -e.b1 : e.t2;
  L.unit = r == 1;
  L.dirx = dir == 1;
  return L;
}
__device__ __forceinline__ void left(const Eig& e, int dir, const double* q, double* c) {
  const fp qf[4] = {q[0], q[1], q[2], q[3]};
  fp cf[4];
  left(e, dir, qf, cf);
#pragma unroll
  for (int k = 0; k < 4; ++k) c[k] = cf[k].v;
}

// R * c (rightEigenVectorx/y, :100-131, 169-180)
__device__ __forceinline__ void right(const Eig& e, int dir, const fp* c, fp* q) {
  fp s = c[0]; s = s + c[2]; s = s + c[3]; q[0] = s;
  if (dir == 1) {
    s = (e.vxm - e.cm) * c[0]; s = s + e.vxm * c[2]; s = s + (e.vxm + e.cm) * c[3]; q[1] = s;
    s = e.vym * c[0]; s = s + c[1]; s = s + e.vym * c[2]; s = s + e.vym * c[3]; q[2] = s;
    s = (e.hm - e.t0r) * c[0]; s = s + e.vym * c[1]; s = s + e.qm * c[2]; s = s + (e.hm + e.t0r) * c[3]; q[3] = s;
  } else {
    s = e.vxm * c[0]; s = s + c[1]; s = s + e.vxm * c[2]; s = s + e.vxm * c[3]; q[1] = s;
    s = (e.vym - e.cm) * c[0]; s = s + e.vym * c[2]; s = s + (e.vym + e.cm) * c[3]; q[2] = s;
    s = (e.hm - e.t0r) * c[0]; s = s + e.vxm * c[1]; s = s + e.qm * c[2]; s = s + (e.hm + e.t0r) * c[3]; q[3] = s;
  }
}

// One side of the HLLC flux (Equations_Euler2D.cpp:372-428): primitives, enthalpy, sound speed.
struct HllcSide {
  fp q[4], w[4], h, c;
};
__device__ __forceinline__ HllcSide hllc_side(double g1, const fp* q, const Den& rho) {
  HllcSide s;
#pragma unroll
  for (int k = 0; k < 4; ++k) s.q[k] = q[k];
  primitive(g1, q, rho, s.w);
  s.h = quot(q[3] + s.w[3], rho);
  s.c = sqrt_abs(quot(s.w[3], rho));
  return s;
}
// The flux from its two sides; rl: the left density
__device__ __forceinline__ void hllc(double g1, int dir, const HllcSide& l, const HllcSide& r, const Den& rl, fp* F) {
  const int d1 = dir - 1;
  fp fl[4], qs[4];
  const fp rr = sqrt_abs(quot(r.w[0], rl));
  const fp rrr = lit(kOne) / (lit(kOne) + rr);
  fp vm[2];
  vm[0] = (l.w[1] + r.w[1] * rr) * rrr;
  vm[1] = (l.w[2] + r.w[2] * rr) * rrr;
  const fp qm = lit(kHalf) * (vm[0] * vm[0] + vm[1] * vm[1]);
  const fp hm = (l.h + r.h * rr) * rrr;
  const fp cm = sqrt_abs(fp(g1) * (hm - qm));
  const fp sl = fmin((l.w[dir] - l.c).v, (vm[d1] - cm).v);
  const fp sr = fmax((r.w[dir] + r.c).v, (vm[d1] + cm).v);
  const fp dl = sl - l.w[dir], dr = sr - r.w[dir];
  const fp sm = (r.q[dir] * dr - l.q[dir] * dl + l.w[3] - r.w[3]) / (r.w[0] * dr - l.w[0] * dl);
  const fp ps = l.w[3] + l.w[0] * (l.w[dir] - sl) * (l.w[dir] - sm);
  // The reference's four regions (:408-427).  The two star regions run the same expressions on
  // the left or the right operands (the energy term keeps the left pressure in both, as the
  // reference does), and so do the two outer regions, so the operands are selected first and
  // one copy of the arithmetic runs: a warp whose faces fall in different regions does not pay
  // for both.  Same operations in the same order on the same values: the same bits.
  const bool outer_l = sl.v > 0.0;
  const bool star_l = !outer_l && sl.v <= 0.0 && sm.v > 0.0;
  const bool star_r = !outer_l && !star_l && sm.v <= 0.0 && sr.v >= 0.0;
  const bool use_l = outer_l || star_l;
  fp q[4], w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    q[k] = use_l ? l.q[k] : r.q[k];
    w[k] = use_l ? l.w[k] : r.w[k];
  }
  flux(dir, q, w, fl);
  if (star_l || star_r) {
    const fp s = use_l ? sl : sr;
    const fp nom = use_l ? dl : dr;
    const Den den = den_of(s - sm);
    qs[0] = quot(w[0] * nom, den);
    qs[1] = quot(dir == 1 ? nom * q[1] + ps - w[3] : nom * q[1], den);
    qs[2] = quot(dir == 2 ? nom * q[2] + ps - w[3] : nom * q[2], den);
    qs[3] = quot(nom * q[3] - l.w[3] * w[dir] + ps * sm, den);
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = fl[k] + s * (qs[k] - q[k]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = fl[k];
  }
}
__device__ __forceinline__ void hllc(double g1, int dir, const fp* ql, const fp* qr, fp* F) {
  const Den rl = den_of(ql[0]);
  hllc(g1, dir, hllc_side(g1, ql, rl), hllc_side(g1, qr, den_of(qr[0])), rl, F);
}

// The two sides of a Gauss point with what the Rusanov fluxes share: primitives, the densities as
// shared denominators, and maxLocalWaveSpeed (:221-246), the four characteristic speeds' maxima.
struct Sides {
  fp wl[4], wr[4], a[4];
  Den rl, rg;
};
__device__ __forceinline__ Sides sides_of(double g, double g1, int dir, const fp* ql, const fp* qr) {
  Sides s;
  s.rl = den_of(ql[0]);
  s.rg = den_of(qr[0]);
  primitive(g1, ql, s.rl, s.wl);
  primitive(g1, qr, s.rg, s.wr);
  const fp cl = sqrt_abs(quot(fp(g) * s.wl[3], s.rl));
  const fp cr = sqrt_abs(quot(fp(g) * s.wr[3], s.rg));
  const fp vl = s.wl[dir], vr = s.wr[dir];
  s.a[0] = max_(abs_(vl - cl), abs_(vr - cr));
  s.a[1] = max_(abs_(vl), abs_(vr));
  s.a[2] = s.a[1];
  s.a[3] = max_(abs_(vl + cl), abs_(vr + cr));
  return s;
}
// (fl + fr - R (a * L (xr - xl))) / 2
__device__ __forceinline__ void dissipate(int dir, const Eig& e, const fp* a, const fp* xl, const fp* xr,
                                          const fp* fl, const fp* fr, fp* F) {
  fp d[4], m[4], rm[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) d[k] = xr[k] - xl[k];
  left(e, dir, d, m);
#pragma unroll
  for (int k = 0; k < 4; ++k) m[k] = a[k] * m[k];
  right(e, dir, m, rm);
#pragma unroll
  for (int k = 0; k < 4; ++k) F[k] = lit(kHalf) * (fl[k] + fr[k] - rm[k]);
}

// characteristic Rusanov (:310-330)
__device__ __forceinline__ void rusanov(int dir, const Eig& e, const Sides& s, const fp* ql, const fp* qr, fp* F) {
  fp fl[4], fr[4];
  flux(dir, ql, s.wl, fl);
  flux(dir, qr, s.wr, fr);
  dissipate(dir, e, s.a, ql, qr, fl, fr, F);
}

// maxSpeed over both directions (Equations_Euler2D.cpp:207-219)
__device__ __forceinline__ double max_speed2(double g, const double* w) {
  const fp c = sqrt_abs(fp(g) * w[3] / w[0]);
  return fmax(fmax((fp(w[1]) - c).v, fabs((fp(w[1]) + c).v)), fmax((fp(w[2]) - c).v, fabs((fp(w[2]) + c).v)));
}

// ---- Equations::Euler1D (Equations_Euler1D.cpp) --------------------------------------------

__device__ __forceinline__ void primitive1(double g1, const fp* q, const Den& d, fp* w) {  // :18-23
  w[0] = q[0];
  w[1] = quot(q[1], d);
  w[2] = (q[2] - lit(kHalf) * q[1] * w[1]) * g1;  // (the half beside the quotient's chain)
}

// eigen1DEuler (FV_System1D.cpp:121-156), eigenvectors :55-89 as full row-major 3x3 matrices
__device__ __forceinline__ void eig1(double g1, fp sra, fp ua, fp ha, fp srb, fp ub, fp hb, fp* R, fp* L) {
  const fp one = lit(kOne), half = lit(kHalf), nhalf = lit(kNegHalf);
  fp t0 = sra / (sra + srb);
  const fp t1 = one - t0;
  const fp vxm = t0 * ua + t1 * ub;
  const fp hm = t0 * ha + t1 * hb;
  const fp qm = half * vxm * vxm;
  const fp cm = sqrt_abs(fp(g1) * (hm - qm));
  t0 = vxm * cm;
  R[0] = one; R[1] = one; R[2] = one;
  R[3] = vxm - cm; R[4] = vxm; R[5] = vxm + cm;
  R[6] = hm - t0; R[7] = qm; R[8] = hm + t0;
  const fp rcm = one / cm;
  const fp b1 = fp(g1) * rcm * rcm;
  const fp b2 = qm * b1;
  const fp s0 = vxm * rcm;
  const fp s1 = b1 * vxm;
  const fp t2 = half * b1;
  L[0] = half * (b2 + s0); L[1] = nhalf * (s1 + rcm); L[2] = t2;
  L[3] = one - b2; L[4] = s1; L[5] = -b1;
  L[6] = half * (b2 - s0); L[7] = nhalf * (s1 - rcm); L[8] = t2;
}

__device__ __forceinline__ void mv3(const fp* M, const fp* x, fp* y) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    fp s = M[3 * i] * x[0];
    s = s + M[3 * i + 1] * x[1];
    s = s + M[3 * i + 2] * x[2];
    y[i] = s;
  }
}

__device__ __forceinline__ void flux1(const fp* q, const fp* w, fp* f) {
  f[0] = q[1];
  f[1] = q[1] * w[1] + w[2];
  f[2] = w[1] * (q[2] + w[2]);
}

// The 1D counterpart of Sides; maxLocalWaveSpeed (Equations_Euler1D.cpp:96-107)
struct Sides1 {
  fp wl[3], wr[3], a[3];
  Den rl, rg;
};
__device__ __forceinline__ Sides1 sides1_of(double g, double g1, const fp* ql, const fp* qr) {
  Sides1 s;
  s.rl = den_of(ql[0]);
  s.rg = den_of(qr[0]);
  primitive1(g1, ql, s.rl, s.wl);
  primitive1(g1, qr, s.rg, s.wr);
  const fp cl = sqrt_abs(quot(fp(g) * s.wl[2], s.rl));
  const fp cr = sqrt_abs(quot(fp(g) * s.wr[2], s.rg));
  s.a[0] = max_(abs_(s.wl[1] - cl), abs_(s.wr[1] - cr));
  s.a[1] = max_(abs_(s.wl[1]), abs_(s.wr[1]));
  s.a[2] = max_(abs_(s.wl[1] + cl), abs_(s.wr[1] + cr));
  return s;
}
__device__ __forceinline__ void dissipate1(const fp* L, const fp* R, const fp* a, const fp* xl, const fp* xr,
                                           const fp* fl, const fp* fr, fp* F) {
  fp d[3], m[3], rm[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) d[k] = xr[k] - xl[k];
  mv3(L, d, m);
#pragma unroll
  for (int k = 0; k < 3; ++k) m[k] = a[k] * m[k];
  mv3(R, m, rm);
#pragma unroll
  for (int k = 0; k < 3; ++k) F[k] = lit(kHalf) * (fl[k] + fr[k] - rm[k]);
}

// Rusanov (Equations_Euler1D.cpp:129-135)
__device__ __forceinline__ void rusanov1(const Sides1& s, const fp* L, const fp* R, const fp* ql, const fp* qr, fp* F) {
  fp fl[3], fr[3];
  flux1(ql, s.wl, fl);
  flux1(qr, s.wr, fr);
  dissipate1(L, R, s.a, ql, qr, fl, fr, F);
}

// One side of the 1D HLLC flux (Equations_Euler1D.cpp:156-210): primitives, enthalpy, sound speed.
struct Hllc1Side {
  fp q[3], w[3], h, c;
};
__device__ __forceinline__ Hllc1Side hllc1_side(double g1, const fp* q, const Den& rho) {
  Hllc1Side s;
#pragma unroll
  for (int k = 0; k < 3; ++k) s.q[k] = q[k];
  primitive1(g1, q, rho, s.w);
  s.h = quot(q[2] + s.w[2], rho);
  s.c = sqrt_abs(quot(s.w[2], rho));
  return s;
}
// The flux from its two sides; rl: the left density.  As in 2D the operands of the left or right
// region are selected first and one copy of the arithmetic runs.
__device__ __forceinline__ void hllc1(double g1, const Hllc1Side& l, const Hllc1Side& r, const Den& rl, fp* F) {
  fp fl[3], qs[3];
  const fp rr = sqrt_abs(quot(r.w[0], rl));
  const fp rrr = lit(kOne) / (lit(kOne) + rr);
  const fp vm = (l.w[1] + r.w[1] * rr) * rrr;
  const fp qm = lit(kHalf) * vm * vm;
  const fp hm = (l.h + r.h * rr) * rrr;
  const fp cm = sqrt_abs(fp(g1) * (hm - qm));
  const fp sl = fmin((l.w[1] - l.c).v, (vm - cm).v);
  const fp sr = fmax((r.w[1] + r.c).v, (vm + cm).v);
  const fp dl = sl - l.w[1], dr = sr - r.w[1];
  const fp sm = (r.q[1] * dr - l.q[1] * dl + l.w[2] - r.w[2]) / (r.w[0] * dr - l.w[0] * dl);
  const fp ps = l.w[2] + l.w[0] * (l.w[1] - sl) * (l.w[1] - sm);
  const bool outer_l = sl.v > 0.0;
  const bool star_l = !outer_l && sl.v <= 0.0 && sm.v > 0.0;
  const bool star_r = !outer_l && !star_l && sm.v <= 0.0 && sr.v >= 0.0;
  const bool use_l = outer_l || star_l;
  fp q[3], w[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    q[k] = use_l ? l.q[k] : r.q[k];
    w[k] = use_l ? l.w[k] : r.w[k];
  }
  flux1(q, w, fl);
  if (star_l || star_r) {
    const fp s = use_l ? sl : sr;
    const fp nom = use_l ? dl : dr;
    const Den den = den_of(s - sm);
    qs[0] = quot(w[0] * nom, den);
    qs[1] = quot(nom * q[1] + ps - w[2], den);
    qs[2] = quot(nom * q[2] - l.w[2] * w[1] + ps * sm, den);
#pragma unroll
    for (int k = 0; k < 3; ++k) F[k] = fl[k] + s * (qs[k] - q[k]);
  } else {
#pragma unroll
    for (int k = 0; k < 3; ++k) F[k] = fl[k];
  }
}
__device__ __forceinline__ void hllc1(double g1, const fp* ql, const fp* qr, fp* F) {
  const Den rl = den_of(ql[0]);
  hllc1(g1, hllc1_side(g1, ql, rl), hllc1_side(g1, qr, den_of(qr[0])), rl, F);
}

__device__ __forceinline__ double max_speed1(double g, fp u, fp p, const Den& rho) {  // :91-94
  const fp c = sqrt_abs(quot(fp(g) * p, rho));
  return fmax(fabs((u - c).v), fabs((u + c).v));
}

// ---- Schemes::Hermite (Schemes_Hermite.cpp) -------------------------------------------------

// smoothnessMeasure (:515-526).  The reference's c0, c1 are twice the sums kept here and its b2
// half of the difference: the factors 4 and 1/4 of their squares are exact and ride in the sum.
__device__ __forceinline__ void hermite_si(const fp* u, const fp* v, fp* SI) {
  const fp u01 = u[0] - u[1], u12 = u[1] - u[2], c1 = lit(kThirteenTwelfths);
  const fp b0 = scaled(kNegTwo, u01, -v[0]), x0 = u01 + v[0];
  const fp b1 = scaled(kNegTwo, u12, -v[2]), x1 = u12 + v[2];
  const fp b2 = u[2] - u[0], x2 = scaled(kNegTwo, u[1], u[0]) + u[2];
  SI[0] = scaled(kFour, c1 * (x0 * x0), b0 * b0);
  SI[1] = scaled(kFour, c1 * (x1 * x1), b1 * b1);
  SI[2] = scaled(kQuarter, b2 * b2, c1 * (x2 * x2));
}
// smoothnessMeasureDerivative (:528-541); c0 and c1 as half the reference's
__device__ __forceinline__ void hermite_sid(const fp* u, const fp* d, fp* SI) {
  const fp c1 = lit(kThirteenTwelfths), six = lit(kSix), three = lit(kThree);
  const fp s01 = six * (u[0] - u[1]), s21 = six * (u[2] - u[1]);
  const fp b0 = scaled(kTwo, scaled(kTwo, d[1], d[0]), s01), x0 = s01 + three * (d[0] + d[1]);
  const fp b1 = scaled(kNegTwo, scaled(kTwo, d[1], d[2]), s21), x1 = three * (d[1] + d[2]) - s21;
  const fp b2 = scaled(kNegTwo, u[1], u[0]) + u[2], x2 = three * (u[2] - u[0]) - six * d[1];
  SI[0] = scaled(kFour, c1 * (x0 * x0), b0 * b0);
  SI[1] = scaled(kFour, c1 * (x1 * x1), b1 * b1);
  SI[2] = c1 * (x2 * x2) + b2 * b2;
}
// fullPointsSI (:597-603)
__device__ __forceinline__ fp hermite_brk(const fp* u, const fp* d) {
  const fp r = (lit(k1029270) * u[2] - lit(k2129184) * u[1] + lit(k1099914) * u[0] + lit(k281121) * d[0] -
                lit(k494958) * d[2]) * d[0] +
               (lit(k2129184) * u[1] - lit(k1029270) * u[0] - lit(k1099914) * u[2] + lit(k281121) * d[2]) * d[2] +
               (lit(k1099445) * u[2] - lit(k4317056) * u[1] + lit(k2118166) * u[0]) * u[2] +
               lit(k4317056) * (u[1] - u[0]) * u[1] + lit(k1099445) * u[0] * u[0];
  return quot_lit(abs_(r), 6720.0, kDiv6720);
}
// fullPointsSId (:605-612)
__device__ __forceinline__ fp hermite_brkd(const fp* u, const fp* d) {
  const fp r = (lit(k3156862) * d[2] + lit(k13189240) * d[1] + lit(k1710479) * d[0] - lit(k9617754) * u[2] -
                lit(k531552) * u[1] + lit(k10149306) * u[0]) * d[0] +
               (lit(k13189240) * d[2] + lit(k26511200) * d[1] - lit(k39700440) * u[2] + lit(k39700440) * u[0]) * d[1] +
               (lit(k1710479) * d[2] - lit(k10149306) * u[2] + lit(k531552) * u[1] + lit(k9617754) * u[0]) * d[2] +
               (lit(k15136011) * u[2] - lit(k1076544) * u[1] - lit(k29195478) * u[0]) * u[2] +
               lit(k1076544) * (u[1] - u[0]) * u[1] + lit(k15136011) * u[0] * u[0];
  return quot_lit(abs_(r), 1680.0, kDiv1680);
}
__device__ __forceinline__ double maxof3(const fp* s) {
  double t = s[0].v;
  t = (t < s[1].v) ? s[1].v : t;
  t = (t < s[2].v) ? s[2].v : t;
  return t;
}
// tau of hteno (full: the full-stencil indicator) or htenoi (improved)
__device__ __forceinline__ double hermite_tau(bool improved, fp full, const fp* SI) {
  if (improved) return maxof3(SI);
  return fabs(scaled(kNegQuarter, scaled(kTwo, SI[2], SI[0] + SI[1]), full).v);
}
// one hteno/htenoi output: cut-off (cutOff/cutOffd, :614-628) and the table weights
__device__ __forceinline__ double hermite_weighted(const DevConst& C, int which, const fp* p,
                                                   const fp* SI, double tau) {
  const int pat = cutoff_pattern(SI, tau, HTENO_HER_CT);
  const double* w = which == 0 ? C.hwtab_m[pat] : which == 1 ? C.hwtab_p[pat]
                  : which == 2 ? C.hwtab_md[pat] : C.hwtab_pd[pat];
  return catchnan(dot3w(p, w).v);
}

// One side of kind 0 hteno (:295-379), 1 htenoi (:670-758) or 2 linear (:760-812) at x_{i+1/2}: side
// 0 from the cells u[0..2], d[0..2] (u^-, d^-), side 1 from the three cells one further to the right
// (u^+, d^+), by the mirrored coefficients in the reference's order.  C in global memory.
__device__ __forceinline__ void hermite_side(const DevConst& C, const HermiteK<double>& K, int kind, const fp* u,
                                             const fp* d, int side, double& val, double& der) {
  auto pick = [&](double c0, double c1) { return fp(side ? c1 : c0); };
  if (kind == 2) {
    fp c[6];
#pragma unroll
    for (int m = 0; m < 5; ++m) c[m] = pick(K.crjlin[m][0], K.crjlin[m][1]);
    val = (dot3(c[0], c[1], c[2], u) + c[3] * d[0] + c[4] * d[2]).v;
#pragma unroll
    for (int m = 0; m < 6; ++m) c[m] = pick(K.crjlind[m][0], K.crjlind[m][1]);
    der = (dot3(c[0], c[1], c[2], u) + dot3(c[3], c[4], c[5], d)).v;
    return;
  }
  const bool imp = kind == 1;
  const fp ud[3] = {d[0] * K.dif, d[1] * K.dif, d[2] * K.dif};
  fp p[3], SI[3];
  const auto& a = K.crj;
  p[0] = pick(a[0][0], a[1][1]) * u[0] + pick(a[1][0], a[0][1]) * u[1] + pick(a[2][0], -a[2][1]) * d[0];
  p[1] = pick(a[0][1], a[1][0]) * u[1] + pick(a[1][1], a[0][0]) * u[2] + pick(a[2][1], -a[2][0]) * d[2];
  p[2] = pick(a[0][2], a[2][2]) * u[0] + fp(a[1][2]) * u[1] + pick(a[2][2], a[0][2]) * u[2];
  hermite_si(u, ud, SI);
  val = hermite_weighted(C, side, p, SI, hermite_tau(imp, imp ? fp(0.0) : hermite_brk(u, ud), SI));

  const auto& b = K.crjd;
  p[0] = pick(b[0][0], b[0][1]) * u[0] + pick(b[1][0], b[1][1]) * u[1] + pick(b[2][0], b[3][1]) * d[0] +
         pick(b[3][0], b[2][1]) * d[1];
  p[1] = pick(b[0][1], b[0][0]) * u[1] + pick(b[1][1], b[1][0]) * u[2] + pick(b[2][1], b[3][0]) * d[1] +
         pick(b[3][1], b[2][0]) * d[2];
  const fp s = pick(b[0][2], b[2][2]) * u[0] + fp(b[1][2]) * u[1] + pick(b[2][2], b[0][2]) * u[2];
  p[2] = (side ? -s : s) + fp(b[3][2]) * d[1];
  hermite_sid(u, ud, SI);
  der = hermite_weighted(C, 2 + side, p, SI, hermite_tau(imp, imp ? fp(0.0) : hermite_brkd(u, ud), SI));
}
// Both sides: out = {u^-, u^+, d^-, d^+}
__device__ __forceinline__ void hermite_recon(const DevConst& C, const HermiteK<double>& K,
                                              int kind, const double* uin, const double* din,
                                              double* out) {
  const fp u[4] = {uin[0], uin[1], uin[2], uin[3]}, d[4] = {din[0], din[1], din[2], din[3]};
  hermite_side(C, K, kind, u, d, 0, out[0], out[2]);
  hermite_side(C, K, kind, u + 1, d + 1, 1, out[1], out[3]);
}

// hermiteLimiter (Schemes_Hermite.cpp:634-662); dif: the cell size, as a shared denominator
__device__ __forceinline__ double hermite_limiter(const Den& dif, const double* uin, const double* din) {
  const fp u[3] = {uin[0], uin[1], uin[2]}, d[3] = {din[0], din[1], din[2]};
  fp p[3], sm[3], w[3];
  p[0] = quot(lit(kThreeQuarters) * (u[2] - u[0]), dif) - lit(kQuarter) * (d[0] + d[2]);
  p[1] = quot(u[1] - u[0], dif);
  p[2] = quot(u[2] - u[1], dif);
  const fp ud[3] = {d[0] * dif.b, d[1] * dif.b, d[2] * dif.b};
  sm[0] = hermite_brk(u, ud);
  sm[1] = (u[0] - u[1]) * (u[0] - u[1]);
  sm[2] = (u[1] - u[2]) * (u[1] - u[2]);
  const fp ta = abs_(sm[0] - sm[1]) + abs_(sm[0] - sm[2]);
  const fp tau = lit(kQuarter) * (ta * ta);
#pragma unroll
  for (int k = 0; k < 3; ++k)
    w[k] = lit(k == 0 ? kLw0 : kLw1) * (lit(kOne) + tau / (sm[k] + lit(kEps6)));
  const Den ds = den_of((w[0] + w[1]) + w[2]);
#pragma unroll
  for (int k = 0; k < 3; ++k) w[k] = quot(w[k], ds);
  const fp r12 = lit(kLw1OverLw0);
  fp inner = r12 * p[1];
  inner = inner + r12 * p[2];
  fp w12 = w[1] * p[1];
  w12 = w12 + w[2] * p[2];
  return (w[0] * (quot(p[0], den_lit(1.0 - 2E-5, kRcpLw0)) - inner) + w12).v;
}
__device__ __forceinline__ double hermite_limiter(const HermiteK<double>& K, const double* u, const double* d) {
  return hermite_limiter(den_of(K.dif), u, d);
}

// A(q) * x with the Jacobians dfluxx / dfluxy (Equations_Euler2D.cpp:52-98), row sums left to
// right; zero and unit entries as in the reference's matrices.
__device__ __forceinline__ void dflux_apply(fp g, fp g1, fp g3, int dir, const fp* q, const fp* w,
                                            const Den& rho, const fp* x, fp* y) {
  const fp half = lit(kHalf);
  if (dir == 1) {
    const fp sv = w[1] * w[1];
    const fp dv = half * g1 * (sv + w[2] * w[2]);
    const fp h = quot(q[3] + w[3], rho);
    y[0] = x[1];
    fp s = (dv - sv) * x[0]; s = s + (-g3 * w[1]) * x[1]; s = s + (-g1 * w[2]) * x[2]; s = s + g1 * x[3]; y[1] = s;
    s = (-w[1] * w[2]) * x[0]; s = s + w[2] * x[1]; s = s + w[1] * x[2]; y[2] = s;
    s = ((dv - h) * w[1]) * x[0]; s = s + (h - g1 * sv) * x[1]; s = s + (-g1 * w[1] * w[2]) * x[2];
    s = s + (g * w[1]) * x[3]; y[3] = s;
  } else {
    const fp sv = w[2] * w[2];
    const fp dv = half * g1 * (sv + w[1] * w[1]);
    const fp h = quot(q[3] + w[3], rho);
    y[0] = x[2];
    fp s = (-w[1] * w[2]) * x[0]; s = s + w[2] * x[1]; s = s + w[1] * x[2]; y[1] = s;
    s = (dv - sv) * x[0]; s = s + (-g1 * w[1]) * x[1]; s = s + (-g3 * w[2]) * x[2]; s = s + g1 * x[3]; y[2] = s;
    s = ((dv - h) * w[2]) * x[0]; s = s + (-g1 * w[1] * w[2]) * x[1]; s = s + (h - g1 * sv) * x[2];
    s = s + (g * w[2]) * x[3]; y[3] = s;
  }
}

// dRusanov (Equations_Euler2D.cpp:352-360) as called in FVHermite_System2D.cpp:553-589
__device__ __forceinline__ void drusanov(double g, double g1, double g3, int dir, const Eig& e, const Sides& s,
                                         const fp* ql, const fp* qr, const fp* dql, const fp* dqr, fp* F) {
  fp al[4], ar[4];
  dflux_apply(g, g1, g3, dir, ql, s.wl, s.rl, dql, al);
  dflux_apply(g, g1, g3, dir, qr, s.wr, s.rg, dqr, ar);
  dissipate(dir, e, s.a, dql, dqr, al, ar, F);
}

// dflux 1D (Equations_Euler1D.cpp:39-53) applied to x; dRusanov 1D (:212-220)
__device__ __forceinline__ void drusanov1(double g, double g1, double g3, const Sides1& s, const fp* L, const fp* R,
                                          const fp* ql, const fp* qr, const fp* dql, const fp* dqr, fp* F) {
  fp al[3], ar[3];
  auto apply = [&](const fp* q, const fp* w, const Den& rho, const fp* x, fp* y) {
    const fp G(g), G1(g1), G3(g3);
    const fp a3 = lit(kHalf) * G3 * w[1] * w[1];
    const fp a4 = -G3 * w[1];
    const fp e = quot(G * q[2], rho);
    const fp a6 = (G1 * (w[1] * w[1]) - e) * w[1];
    const fp a7 = e - lit(kThreeHalves) * G1 * w[1] * w[1];
    const fp a8 = G * w[1];
    y[0] = x[1];
    fp t = a3 * x[0]; t = t + a4 * x[1]; t = t + G1 * x[2]; y[1] = t;
    t = a6 * x[0]; t = t + a7 * x[1]; t = t + a8 * x[2]; y[2] = t;
  };
  apply(ql, s.wl, s.rl, dql, al);
  apply(qr, s.wr, s.rg, dqr, ar);
  dissipate1(L, R, s.a, dql, dqr, al, ar, F);
}

}  // namespace par
}  // namespace hteno
