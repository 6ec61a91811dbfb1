// Packed pieces (f32x2.cuh) that the mixed FV 2D and Hermite 2D kernels share: GL3 of both sides of a
// face, the Roe projection of two cells, the back-projection of both sides.  Each half gets the bits of
// the scalar function of device_math.cuh or hermite_math.cuh, which the pointwise entry points run
// (tests/cuda/packed_pairs.cu compares them).
#pragma once

#include "device_math.cuh"
#include "f32x2.cuh"
#include "hermite_math.cuh"

namespace hteno {

// A constant pair of DevConst.
__device__ __forceinline__ f2 cpair(const float (&p)[2]) { return pack(p[0], p[1]); }

__device__ __forceinline__ f2 rcp2(f2 x) { return pack(Cst<float>::rcp(lo(x)), Cst<float>::rcp(hi(x))); }
__device__ __forceinline__ f2 max2(f2 a, f2 b) { return pack(fmaxf(lo(a), lo(b)), fmaxf(hi(a), hi(b))); }
__device__ __forceinline__ f2 catchnan2(f2 x) { return pack(catchnan(lo(x)), catchnan(hi(x))); }
// x0 y0 + x1 y1, the first product fused
__device__ __forceinline__ f2 dot2m(f2 x0, f2 y0, f2 x1, f2 y1) { return mad(x0, y0, x1 * y1); }

// p0 w0 + p1 w1 + p2 w2 with the weights of the cut-off patterns (teno_pattern of device_math.cuh) that the
// ratios 1 + tau / (S_k + epsz) give, one per half; tm, tp: the two halves' tables.  The lane's products
// are summed in the order k = 0 fused on 1, then 2 (kFirst), or left to right.
template <bool kFirst>
__device__ __forceinline__ f2 cutoff_sum(f2 p0, f2 p1, f2 p2, f2 S0, f2 S1, f2 S2, f2 tau, float ct,
                                         const float (*tm)[3], const float (*tp)[3]) {
  const f2 ez = dup(HTENO_F32_EPSZ), one = dup(1.0f);
  const f2 r0 = mad(tau, rcp2(S0 + ez), one), r1 = mad(tau, rcp2(S1 + ez), one), r2 = mad(tau, rcp2(S2 + ez), one);
  const f2 inv = rcp2(max2(max2(r0, r1), r2));
  auto sixth = [](f2 x) {
    const f2 q = x * x;
    return q * q * q;
  };
  const f2 e0 = sixth(r0 * inv), e1 = sixth(r1 * inv), e2 = sixth(r2 * inv);
  const f2 lim = dup(ct) * ((e0 + e1) + e2);
  auto pattern = [](float a0, float a1, float a2, float l) {
    return (a0 < l ? 0 : 1) | (a1 < l ? 0 : 2) | (a2 < l ? 0 : 4);
  };
  const float* wm = tm[pattern(lo(e0), lo(e1), lo(e2), lo(lim))];
  const float* wp = tp[pattern(hi(e0), hi(e1), hi(e2), hi(lim))];
  const f2 w0 = pack(wm[0], wp[0]), w1 = pack(wm[1], wp[1]), w2 = pack(wm[2], wp[2]);
  return catchnan2(kFirst ? mad(p2, w2, dot2m(p0, w0, p1, w1)) : dot3m(p0, w0, p1, w1, p2, w2));
}

// Tables of a block of the Hermite 2D face kernel, in shared memory (a per-thread pattern would serialise
// constant-memory reads): candidate coefficients of both sides (cu of the value, cd of the derivative)
// and the weights per cut-off pattern of HTENO (value -, +, derivative -, +) and TENO5 (-, +).
struct HermiteTab {
  f2 cu[3][3], cd[3][4];
  float hw[4][8][3], lw[2][8][3];
};
// The whole block calls it.
__device__ __forceinline__ void load_hermite_tab(HermiteTab& S, const HermiteK<float>& K, const DevConst& C) {
  for (int e = threadIdx.x; e < 96; e += blockDim.x) {
    (&S.hw[0][0][0])[e] = Cst<float>::hwtab(C, e / 24, e / 3 % 8)[e % 3];
    if (e < 48) (&S.lw[0][0][0])[e] = Cst<float>::wtab(C, e / 24, e / 3 % 8)[e % 3];
  }
  if (threadIdx.x == 0) {
    const float (&a)[3][3] = K.crj, (&b)[4][3] = K.crjd;
    // (candidate k: two cell values and a derivative, or three cell values)
    S.cu[0][0] = pack(a[0][0], a[1][1]); S.cu[0][1] = pack(a[1][0], a[0][1]); S.cu[0][2] = pack(a[2][0], -a[2][1]);
    S.cu[1][0] = pack(a[0][1], a[1][0]); S.cu[1][1] = pack(a[1][1], a[0][0]); S.cu[1][2] = pack(a[2][1], -a[2][0]);
    S.cu[2][0] = pack(a[0][2], a[2][2]); S.cu[2][1] = pack(a[1][2], a[1][2]); S.cu[2][2] = pack(a[2][2], a[0][2]);
    // (two cell values and two derivatives; three cell values and the middle derivative)
    S.cd[0][0] = pack(b[0][0], b[0][1]); S.cd[0][1] = pack(b[1][0], b[1][1]);
    S.cd[0][2] = pack(b[2][0], b[3][1]); S.cd[0][3] = pack(b[3][0], b[2][1]);
    S.cd[1][0] = pack(b[0][1], b[0][0]); S.cd[1][1] = pack(b[1][1], b[1][0]);
    S.cd[1][2] = pack(b[2][1], b[3][0]); S.cd[1][3] = pack(b[3][1], b[2][0]);
    S.cd[2][0] = pack(b[0][2], -b[2][2]); S.cd[2][1] = pack(b[1][2], -b[1][2]);
    S.cd[2][2] = pack(b[2][2], -b[0][2]); S.cd[2][3] = pack(b[3][2], b[3][2]);
  }
  __syncthreads();
}

// HTENO (Schemes_Hermite.cpp:295-379; hermite_recon of hermite_math.cuh, kind 0) of both sides of a face:
// U, V the cell pairs (0, 1), (2, 3) of the averages, A, B of the derivatives.  Every product and sum rounds
// as the compiler contracts the scalar function in a unit where it may: the first of two products is fused,
// in S and on the minus side of brkd's second bracket the other one.
struct HtenoSides {
  f2 u, d;  // (minus, plus) values and derivatives
};
__device__ __forceinline__ HtenoSides hteno_sides(const HermiteTab& T, float dif, f2 U, f2 V, f2 A, f2 B) {
  HtenoSides o;
  const f2 u0 = U, u1 = pack(hi(U), lo(V)), u2 = V;  // cells 0..2 for the minus side, 1..3 for the plus side
  const f2 d0 = A, d1 = pack(hi(A), lo(B)), d2 = B;
  const f2 h = dup(dif), v0 = d0 * h, v1 = d1 * h, v2 = d2 * h;
  const f2 m2 = dup(-2.0f), two = dup(2.0f), six = dup(6.0f), c13 = dup(float(HTENO_C1)), quarter = dup(0.25f);
  const f2 u01 = u0 - u1, u12 = u1 - u2, u10 = u1 - u0, u20 = u2 - u0;
  const f2 second = mad(m2, u1, u0) + u2;
  auto indicator = [&](f2 b, f2 c) { return mad(b, b, c13 * c * c); };
  {
    const f2 S0 = indicator(mad(m2, u01, -v0), m2 * (u01 + v0));
    const f2 S1 = indicator(mad(m2, u12, -v2), mad(two, u12, two * v2));
    const f2 S2 = indicator(u20 * dup(0.5f), second);
    const f2 t1 = mad(dup(-494958.0f), v2, mad(dup(281121.0f), v0, mad(dup(1099914.0f), u0,
                      dot2m(dup(1029270.0f), u2, dup(-2129184.0f), u1))));
    const f2 t2 = mad(dup(281121.0f), v2, mad(dup(-1099914.0f), u2, dot2m(dup(-1029270.0f), u0, dup(2129184.0f), u1)));
    const f2 t3 = mad(dup(2118166.0f), u0, dot2m(dup(1099445.0f), u2, dup(-4317056.0f), u1));
    f2 s = mad(t3, u2, dot2m(t1, v0, t2, v2));
    s = mad(dup(1099445.0f) * u0, u0, mad(dup(4317056.0f) * u10, u1, s));
    const f2 tau = abs_(mad(abs_(s), dup(float(1.0 / 6720.0)), -(quarter * mad(two, S2, S0 + S1))));
    const f2 p0 = mad(T.cu[0][2], d0, dot2m(T.cu[0][0], u0, T.cu[0][1], u1));
    const f2 p1 = mad(T.cu[1][2], d2, dot2m(T.cu[1][0], u1, T.cu[1][1], u2));
    const f2 p2 = mad(T.cu[2][2], u2, dot2m(T.cu[2][0], u0, T.cu[2][1], u1));
    o.u = cutoff_sum<true>(p0, p1, p2, S0, S1, S2, tau, float(HTENO_HER_CT), T.hw[0], T.hw[1]);
  }
  {
    const f2 four = dup(4.0f), twelve = dup(12.0f);
    const f2 S0 = indicator(mad(six, u01, mad(two, v0, four * v1)), dot2m(twelve, u01, six, v0 + v1));
    const f2 S1 = indicator(mad(six, u2 - u1, -mad(four, v1, two * v2)), dot2m(twelve, u12, six, v1 + v2));
    const f2 S2 = indicator(second, dot2m(dup(3.0f), u20, dup(-6.0f), v1));
    const f2 t1 = mad(dup(10149306.0f), u0, mad(dup(-531552.0f), u1, mad(dup(-9617754.0f), u2, mad(dup(1710479.0f), v0,
                      dot2m(dup(3156862.0f), v2, dup(13189240.0f), v1)))));
    const f2 t2 = mad(dup(39700440.0f), u0, mad(dup(-39700440.0f), u2,
                      dot2m(pack(26511200.0f, 13189240.0f), pack(lo(v1), hi(v2)),
                            pack(13189240.0f, 26511200.0f), pack(lo(v2), hi(v1)))));
    const f2 t3 = mad(dup(9617754.0f), u0, mad(dup(531552.0f), u1, dot2m(dup(1710479.0f), v2, dup(-10149306.0f), u2)));
    const f2 t4 = mad(dup(-29195478.0f), u0, dot2m(dup(15136011.0f), u2, dup(-1076544.0f), u1));
    f2 s = mad(t4, u2, mad(t3, v2, dot2m(t1, v0, t2, v1)));
    s = mad(dup(15136011.0f) * u0, u0, mad(dup(1076544.0f) * u10, u1, s));
    const f2 tau = abs_(mad(abs_(s), dup(float(1.0 / 1680.0)), -(quarter * mad(two, S2, S0 + S1))));
    const f2 p0 = mad(T.cd[0][3], d1, mad(T.cd[0][2], d0, dot2m(T.cd[0][0], u0, T.cd[0][1], u1)));
    const f2 p1 = mad(T.cd[1][3], d2, mad(T.cd[1][2], d1, dot2m(T.cd[1][0], u1, T.cd[1][1], u2)));
    const f2 p2 = mad(T.cd[2][3], d1, mad(T.cd[2][2], u2, dot2m(T.cd[2][0], u0, T.cd[2][1], u1)));
    o.d = cutoff_sum<true>(p0, p1, p2, S0, S1, S2, tau, float(HTENO_HER_CT), T.hw[2], T.hw[3]);
  }
  return o;
}

// TENO5 (Schemes_Lagrange.cpp:481-511; lagrange_recon of device_math.cuh, kind 0) of both sides of a face
// from the cell pairs (0, 1), (2, 3), (4, 5), tau's first product fused.
__device__ __forceinline__ f2 teno5_sides(const DevConst& C, const HermiteTab& T, f2 P0, f2 P1, f2 P2) {
  const f2 v0 = P0, v1 = pack(hi(P0), lo(P1)), v2 = P1, v3 = pack(hi(P1), lo(P2)), v4 = P2;
  const f2 m2 = dup(-2.0f), m4 = dup(-4.0f), half = dup(0.5f), c13 = dup(float(HTENO_C1));
  const f2 c0 = mad(m2, v3, v2) + v4, b0 = (mad(m4, v3, dup(3.0f) * v2) + v4) * half;
  const f2 c1 = mad(m2, v2, v1) + v3, b1 = (v1 - v3) * half;
  const f2 c2 = mad(m2, v1, v0) + v2, b2 = mad(dup(3.0f), v2, mad(m4, v1, v0)) * half;
  const f2 S0 = mad(c13 * c0, c0, b0 * b0), S1 = mad(c13 * c1, c1, b1 * b1), S2 = mad(c13 * c2, c2, b2 * b2);
  const f2 a4 = mad(dup(8209.0f), v0, mad(dup(-38947.0f), v1, mad(dup(67923.0f), v2,
                    mad(dup(-51001.0f), v3, dup(6908.0f) * v4))));
  const f2 a3 = mad(dup(-38947.0f), v0, mad(dup(179098.0f), v1, mad(dup(-299076.0f), v2, dup(104963.0f) * v3)));
  const f2 a2 = mad(dup(67923.0f), v0, mad(dup(-299076.0f), v1, dup(231153.0f) * v2));
  const f2 a1 = mad(dup(-51001.0f), v0, dup(104963.0f) * v1);
  const f2 r = mad(dup(6908.0f) * v0, v0, mad(v1, a1, mad(v2, a2, mad(v3, a3, v4 * a4))));
  const f2 mean = mad(dup(4.0f), S1, S0 + S2) * dup(float(1.0 / 6.0));
  const f2 tau = abs_(mad(r, dup(float(1.0 / 5040.0)), -mean));
  const f2 p0 = dot3m(cpair(C.x2_cand[0][0]), v2, cpair(C.x2_cand[0][1]), v3, cpair(C.x2_cand[0][2]), v4);
  const f2 p1 = dot3m(cpair(C.x2_cand[1][0]), v1, cpair(C.x2_cand[1][1]), v2, cpair(C.x2_cand[1][2]), v3);
  const f2 p2 = dot3m(cpair(C.x2_cand[2][0]), v0, cpair(C.x2_cand[2][1]), v1, cpair(C.x2_cand[2][2]), v2);
  return cutoff_sum<false>(p0, p1, p2, S0, S1, S2, tau, float(HTENO_LAG_CT), T.lw[0], T.lw[1]);
}

// GL3 (weno5JS3PointsQuadrature, as gl3() of device_math.cuh) of the left (low half) and right (high
// half) face values of one field at once.  kContract: the difference of the middle point fused, as the
// compiler fuses the scalar one in a unit where it may.
struct Gl3f {
  f2 a, b, c;
};
template <bool kContract>
__device__ __forceinline__ Gl3f gl3_pair(const DevConst& C, f2 u0, f2 u1, f2 u2, f2 u3, f2 u4) {
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
  o.a = catchnan2(cand(C.x2_gp, C.x2_linwp));
  const f2 r24 = dup(1.0f / 24.0f), two = dup(2.0f), t23 = dup(23.0f);
  const f2 q0 = mad(t23, u2, mad(two, u1, -u0)) * r24;
  const f2 q1 = (mad(dup(26.0f), u2, -u1) - u3) * r24;
  const f2 q2 = (mad(two, u3, t23 * u2) - u4) * r24;
  const f2 c = mix(C.x2_linw0p, q0, q1, q2), d = cpair(C.x2_sumw0m) * mix(C.x2_linw0m, q0, q1, q2);
  o.b = catchnan2(kContract ? mad(cpair(C.x2_sumw0p), c, -d) : cpair(C.x2_sumw0p) * c - d);
  o.c = catchnan2(cand(C.x2_gm, C.x2_linwm));
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
