// Packed pieces (f32x2.cuh) that the mixed FV 2D and Hermite 2D kernels share: GL3 of both sides of a
// face, the Roe projection of two cells, the back-projection of both sides.  Each half gets the bits of
// the scalar function of device_math.cuh.
#pragma once

#include "device_math.cuh"
#include "f32x2.cuh"

namespace hteno {

// A constant pair of DevConst.
__device__ __forceinline__ f2 cpair(const float (&p)[2]) { return pack(p[0], p[1]); }

// GL3 (weno5JS3PointsQuadrature, as gl3() of device_math.cuh) of the left (low half) and right (high
// half) face values of one field at once.  kContract: the difference of the middle point fused, as the
// compiler fuses the scalar one in a unit where it may.
struct Gl3f {
  f2 a, b, c;
};
template <bool kContract>
__device__ __forceinline__ Gl3f gl3_pair(const DevConst& C, f2 u0, f2 u1, f2 u2, f2 u3, f2 u4) {
  auto rcp2 = [](f2 x) { return pack(Cst<float>::rcp(lo(x)), Cst<float>::rcp(hi(x))); };
  auto nan2 = [](f2 x) { return pack(catchnan(lo(x)), catchnan(hi(x))); };
  const f2 m2 = dup(-2.0f), m4 = dup(-4.0f), c13 = dup(float(HTENO_C1)), q4 = dup(0.25f), eps = dup(float(HTENO_LAG_EPS));
  const f2 bg0 = mad(dup(3.0f), u2, mad(m4, u1, u0));
  const f2 cg0 = mad(m2, u1, u0) + u2;
  const f2 bg1 = u1 - u3;
  const f2 cg1 = mad(m2, u2, u1) + u3;
  const f2 bg2 = mad(m4, u3, dup(3.0f) * u2) + u4;
  const f2 cg2 = mad(m2, u3, u2) + u4;
  f2 s0 = eps + mad(c13 * cg0, cg0, q4 * bg0 * bg0);
  f2 s1 = eps + mad(c13 * cg1, cg1, q4 * bg1 * bg1);
  f2 s2 = eps + mad(c13 * cg2, cg2, q4 * bg2 * bg2);
  s0 = s0 * s0;
  s1 = s1 * s1;
  s2 = s2 * s2;
  // alpha_k = 1 / s_k, scaled by the smallest s to keep float in range
  const f2 smin = pack(fminf(fminf(lo(s0), lo(s1)), lo(s2)), fminf(fminf(hi(s0), hi(s1)), hi(s2)));
  const f2 a0 = smin * rcp2(s0), a1 = smin * rcp2(s1), a2 = smin * rcp2(s2);
  auto mix = [&](const float (&lw)[3][2], f2 q0, f2 q1, f2 q2) {
    const f2 g0 = cpair(lw[0]) * a0, g1 = cpair(lw[1]) * a1, g2 = cpair(lw[2]) * a2;
    return dot3m(q0, g0, q1, g1, q2, g2) * rcp2(g0 + g1 + g2);
  };
  auto cand = [&](const float (&g)[3][3][2], const float (&lw)[3][2]) {
    const f2 q0 = dot3m(cpair(g[0][0]), u0, cpair(g[0][1]), u1, cpair(g[0][2]), u2);
    const f2 q1 = dot3m(cpair(g[1][0]), u1, cpair(g[1][1]), u2, cpair(g[1][2]), u3);
    const f2 q2 = dot3m(cpair(g[2][0]), u2, cpair(g[2][1]), u3, cpair(g[2][2]), u4);
    return mix(lw, q0, q1, q2);
  };
  Gl3f o;
  o.a = nan2(cand(C.x2_gp, C.x2_linwp));
  const f2 r24 = dup(1.0f / 24.0f), two = dup(2.0f), t23 = dup(23.0f);
  const f2 q0 = mad(t23, u2, mad(two, u1, -u0)) * r24;
  const f2 q1 = (mad(dup(26.0f), u2, -u1) - u3) * r24;
  const f2 q2 = (mad(two, u3, t23 * u2) - u4) * r24;
  const f2 c = mix(C.x2_linw0p, q0, q1, q2), d = cpair(C.x2_sumw0m) * mix(C.x2_linw0m, q0, q1, q2);
  o.b = nan2(kContract ? mad(cpair(C.x2_sumw0p), c, -d) : cpair(C.x2_sumw0p) * c - d);
  o.c = nan2(cand(C.x2_gm, C.x2_linwm));
  return o;
}

// Roe projection L q of two cells at once (roe_left of device_math.cuh): q[v] the cells' pair of
// conserved variable v, c[r] their pair of characteristic field r.
struct LeftRows {
  f2 t2, tvt, n0, d0, nvt, nb1, bvt, s1, d2, n3, d3;
};
__device__ __forceinline__ LeftRows left_rows(const Roe2<float>& s, int dir) {
  const float vn = dir == 1 ? s.vxm : s.vym, vt = dir == 1 ? s.vym : s.vxm;
  const float b2 = s.qm * s.b1, s0 = vn * s.rcm, s1 = s.b1 * vn, t2 = 0.5f * s.b1;
  LeftRows L;
  L.t2 = dup(t2);
  L.tvt = dup(-t2 * vt);
  L.n0 = dup(-0.5f * (s1 + s.rcm));
  L.d0 = dup(0.5f * (b2 + s0));
  L.nvt = dup(-vt);
  L.nb1 = dup(-s.b1);
  L.bvt = dup(s.b1 * vt);
  L.s1 = dup(s1);
  L.d2 = dup(1.0f - b2);
  L.n3 = dup(-0.5f * (s1 - s.rcm));
  L.d3 = dup(0.5f * (b2 - s0));
  return L;
}
__device__ __forceinline__ void project2(const LeftRows& L, int dir, const f2* q, f2* c) {
  const f2 qn = dir == 1 ? q[1] : q[2], qt = dir == 1 ? q[2] : q[1];
  c[0] = mad(L.t2, q[3], mad(L.tvt, qt, mad(L.n0, qn, L.d0 * q[0])));
  c[1] = mad(L.nvt, q[0], qt);
  c[2] = mad(L.nb1, q[3], mad(L.bvt, qt, mad(L.s1, qn, L.d2 * q[0])));
  c[3] = mad(L.t2, q[3], mad(L.tvt, qt, mad(L.n3, qn, L.d3 * q[0])));
}

// R c of two characteristic vectors at once (roe_right of device_math.cuh).
__device__ __forceinline__ void right2(const Roe2<float>& s, int dir, const f2* c, f2* q) {
  const float vn = dir == 1 ? s.vxm : s.vym, vt = dir == 1 ? s.vym : s.vxm, t0 = vn * s.cm;
  q[0] = c[0] + c[2] + c[3];
  const f2 qn = mad(dup(vn + s.cm), c[3], mad(dup(vn), c[2], dup(vn - s.cm) * c[0]));
  const f2 qt = mad(dup(vt), c[3], mad(dup(vt), c[2], mad(dup(vt), c[0], c[1])));
  q[dir == 1 ? 1 : 2] = qn;
  q[dir == 1 ? 2 : 1] = qt;
  q[3] = mad(dup(s.hm + t0), c[3], mad(dup(s.qm), c[2], mad(dup(vt), c[1], dup(s.hm - t0) * c[0])));
}

}  // namespace hteno
