// One cell of the Hermite limiter (hermiteLimiter, Schemes_Hermite.cpp:634-662) as a Gauss-Seidel
// sweep along a line sees it, shared by the 1D and 2D Hermite solvers.
#pragma once

#include "hermite_math.cuh"
#include "mixed_conv.cuh"
#include "parity_math.cuh"

namespace hteno {

// Equality of two values' bits (a NaN equals itself, +0 and -0 differ).
__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// One cell of hermiteLimiter (Schemes_Hermite.cpp:634-662) as a sweep from left to right sees it:
// next() takes the right neighbour's average and (unlimited) moment, at() the left neighbour's
// limited moment.  What the next cell shares with this one is carried over.
template <typename T>
struct LimitSweep;

// Double: par::hermite_limiter's operations (the same bits); the difference quotient, its square
// and the latter's reciprocal to the left of a cell are those to the right of the cell before.
template <>
struct LimitSweep<double> {
  par::Den dif, r1, r2;  // r_k: s_k + eps
  par::fp u0, u1, u2, d2, p1, p2, s1, s2;
  __device__ __forceinline__ LimitSweep(const HermiteK<double>& K, double ul, double uc)
      : dif(par::den_of(K.dif)), u1(ul), u2(uc) {
    flat_ok = false;
    right();
  }
  __device__ __forceinline__ void right() {
    p2 = par::quot(u2 - u1, dif);
    s2 = (u1 - u2) * (u1 - u2);
    r2 = par::den_of(s2 + par::lit(par::kEps6));
  }
  __device__ __forceinline__ void next(double ur, double dr) {
    u0 = u1;
    u1 = u2;
    p1 = p2;
    s1 = s2;
    r1 = r2;
    u2 = ur;
    d2 = dr;
    if (!(flat_ok && same_bits(u0.v, u1.v) && same_bits(u1.v, u2.v))) right();  // else p2, s2, r2 stay
  }
  // A cell on constant data with a zero moment to its right (a tail running out into a flat region:
  // the limited moment there shrinks by a quarter per cell for hundreds of cells): every operand but
  // d0 is the flat value's, so the weights are those of the cell before if the full-stencil
  // indicator before its scaling, r, has the same bits -- or is below 5e-21 in both cells, where
  // s0 = r / 6720 < 1e-24 is lost in s0 + 1e-6 and tau = s0^2 in 1 + tau / 1e-6 -- and the terms in
  // p1, p2 are +0.  13 operations instead of ~100.
  bool flat_ok;
  par::fp flat_u, flat_a, flat_z, flat_v, flat_r, flat_w;
  __device__ __forceinline__ bool flat() const {
    return same_bits(u0.v, u1.v) && same_bits(u1.v, u2.v) && same_bits(d2.v, 0.0);
  }
  __device__ __forceinline__ double at_flat(double dl) {
    using namespace par;
    const fp d0(dl);
    if (!flat_ok || !same_bits(flat_u.v, u1.v)) {
      flat_u = u1;
      flat_a = lit(k1029270) * u1 - lit(k2129184) * u1 + lit(k1099914) * u1;
      flat_z = (lit(k1099445) * u1 - lit(k4317056) * u1 + lit(k2118166) * u1) * u1;
      flat_v = lit(k1099445) * u1 * u1;
      flat_ok = true;
      flat_r = flat_indicator(d0);
      const double lim = at(dl, &flat_w);
      return lim;
    }
    const fp r = flat_indicator(d0);
    if (!same_bits(r.v, flat_r.v) && !(r.v < 5e-21 && flat_r.v < 5e-21)) {
      flat_r = r;
      return at(dl, &flat_w);
    }
    const fp p0 = fp(0.0) - lit(kQuarter) * (d0 + d2);
    return (flat_w * quot(p0, den_lit(1.0 - 2E-5, kRcpLw0)) + fp(0.0)).v;
  }
  // |hermite_brk|'s sum on flat data: the terms left out are zeros
  __device__ __forceinline__ par::fp flat_indicator(par::fp d0) const {
    const par::fp ud0 = d0 * dif.b;
    return par::abs_((flat_a + par::lit(par::k281121) * ud0) * ud0 + flat_z + flat_v);
  }
  __device__ __forceinline__ double at(double dl, par::fp* w0n = nullptr) const {
    using namespace par;
    const fp d0(dl), u[3] = {u0, u1, u2}, ud[3] = {d0 * dif.b, fp(0.0), d2 * dif.b};
    const fp p0 = quot(lit(kThreeQuarters) * (u2 - u0), dif) - lit(kQuarter) * (d0 + d2);
    const fp s0 = hermite_brk(u, ud);
    const fp ta = abs_(s0 - s1) + abs_(s0 - s2), t4 = ta * ta;  // tau = t4 / 4: the factor is exact
    const fp one = lit(kOne);
    fp w0 = lit(kLw0) * scaled(kQuarter, quot(t4, den_of(s0 + lit(kEps6))), one);
    fp w1 = lit(kLw1) * scaled(kQuarter, quot(t4, r1), one);
    fp w2 = lit(kLw1) * scaled(kQuarter, quot(t4, r2), one);
    const Den ds = den_of((w0 + w1) + w2);
    w0 = quot(w0, ds);
    w1 = quot(w1, ds);
    w2 = quot(w2, ds);
    if (w0n) *w0n = w0;
    const fp r12 = lit(kLw1OverLw0);
    const fp inner = r12 * p1 + r12 * p2;
    const fp w12 = w1 * p1 + w2 * p2;
    return (w0 * (quot(p0, den_lit(1.0 - 2E-5, kRcpLw0)) - inner) + w12).v;
  }
};

// Float: restated so that little waits for the left neighbour's limited value d0.  hermiteLimiter's
// result is
//   lim = [w0 (p0/lw0 - Q) + w1 p1 + w2 p2] / (w0 + w1 + w2),  w_k = lw_k (1 + tau / (s_k + eps))
// where only p0 = P - d0/4 and s0 = |(a ud0 + B) ud0 + C|/6720 (ud0 = d0 dif, the smoothness
// measure fullPointsSI expanded in ud0) depend on d0.  next() computes B, C, s1, s2, E = P/lw0 - Q,
// M = lw1 r1 + lw2 r2, L = lw1 p1 + lw2 p2, N = lw1 r1 p1 + lw2 r2 p2 with r_k = 1/(s_k + eps); at()
//   tau = (|s0 - s1| + |s0 - s2|)^2 / 4,  w0 = lw0 (1 + tau / (s0 + eps)),
//   lim = (w0 (E - d0 / (4 lw0)) + L + tau N) / (w0 + lw1 + lw2 + tau M).
template <>
struct LimitSweep<float> {
  static constexpr float lw0 = 1.0f - 2e-5f, lw1 = 1e-5f, lw2 = 1e-5f, eps = float(HTENO_LAG_EPS);
  float dif, rdif, u0, u1, u2, B, Cc, p1, p2, r1, r2, s1, s2, E, M, L, N;
  template <typename T>
  __device__ __forceinline__ LimitSweep(const HermiteK<T>& K, float ul, float uc)
      : dif(float(K.dif)), rdif(float(K.rdif)), u1(ul), u2(uc) {
    right();
  }
  __device__ __forceinline__ void right() {
    p2 = (u2 - u1) * rdif;
    s2 = (u1 - u2) * (u1 - u2);
    r2 = 1.0f / (s2 + eps);
  }
  __device__ __forceinline__ void next(float ur, float dr) {
    u0 = u1;
    u1 = u2;
    u2 = ur;
    const float ud2 = dr * dif;
    p1 = p2;
    s1 = s2;
    r1 = r2;
    right();
    constexpr float k6720 = 1.0f / 6720.0f;
    B = (1029270.0f * u2 - 2129184.0f * u1 + 1099914.0f * u0 - 494958.0f * ud2) * k6720;
    Cc = ((-1029270.0f * u0 + 2129184.0f * u1 - 1099914.0f * u2 + 281121.0f * ud2) * ud2 +
          (1099445.0f * u2 - 4317056.0f * u1 + 2118166.0f * u0) * u2 +
          4317056.0f * (u1 - u0) * u1 + 1099445.0f * u0 * u0) * k6720;
    const float P = 0.75f * (u2 - u0) * rdif - 0.25f * dr;
    E = P * (1.0f / lw0) - ((lw1 / lw0) * p1 + (lw2 / lw0) * p2);
    M = lw1 * r1 + lw2 * r2;
    L = lw1 * p1 + lw2 * p2;
    N = lw1 * r1 * p1 + lw2 * r2 * p2;
  }
  __device__ __forceinline__ float at(float d0) const {
    constexpr float a = 281121.0f / 6720.0f, c4 = 0.25f / lw0;
    const float ud0 = d0 * dif;
    const float s0 = fabsf(fmaf(fmaf(a, ud0, B), ud0, Cc));
    const float t = fabsf(s0 - s1) + fabsf(s0 - s2);
    const float tau = 0.25f * t * t;
    const float w0 = lw0 * fmaf(tau, __fdividef(1.0f, s0 + eps), 1.0f);
    const float num = fmaf(w0, fmaf(-c4, d0, E), fmaf(tau, N, L));
    const float den = w0 + fmaf(tau, M, lw1 + lw2);
    return __fdividef(num, den);
  }
};

}  // namespace hteno
