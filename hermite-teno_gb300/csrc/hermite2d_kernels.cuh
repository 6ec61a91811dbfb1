// Kernels of FVHermite::System2D, templated on the compute type.  Included by hermite2d.cu
// (float instantiation, fused multiply-adds allowed) and hermite2d_fp64.cu (double
// instantiation, compiled with --fmad=false and routed through the bit-reproducible
// parity functions).  Each including translation unit owns its constant block.
#pragma once

#include <algorithm>
#include <type_traits>

#include "hermite_limit.cuh"
#include "hteno_internal.h"
#include "limit_rule.h"
#include "mixed_pairs.cuh"

namespace hteno {

constexpr int kHFaceThreads = 128;
constexpr int kHFluxThreads = 64;
// Blocks per SM that the face kernel's registers are cut for: in float 5, 6, 7 blocks (96, 80, 72
// registers, a few spilled) took 413, 408, 405 us at 2048^2, unbounded 130-136.
template <typename T> constexpr int kHFaceBlocks = std::is_same<T, float>::value ? 7 : 1;

struct GeoH {
  int nx, ny;
  double dx, dy, area, gamma, g1, g3;  // g3 = gamma - 3 as the reference computes it
  double rdx, rdy;                     // 1/dx, 1/dy
  float rdxf, rdyf;                    // the same in float (mixed-precision update)
};

// Loads of the double state into the compute type and back: for float on the integer pipes
// (mix::d2f / f2d), for double the identity.
template <typename T>
__device__ __forceinline__ T from_d(double x) {
  if constexpr (std::is_same<T, float>::value) return mix::d2f(x);
  else return x;
}
template <typename T>
__device__ __forceinline__ double to_d(T x) {
  if constexpr (std::is_same<T, float>::value) return mix::f2d(x);
  else return x;
}

template <typename T>
struct WorkH {
  double* prim;   // [4][nc] u, v, h, sqrt|rho| (double)
  T* xc;          // [24][ny][nx+1]: kind a (0 u-, 1 u+, 2 vn-, 3 vn+, 4 vt-, 5 vt+) x field r
  T* xroe;        // [7][ny][nx+1]
  T* yc;          // [24][ny+1][nx]
  T* yroe;        // [7][ny+1][nx]
  T* fx;          // [12][ny][nx+1]: kind (0 u, 1 moment along the sweep, 2 cross moment) x field
  T* fy;          // [12][ny+1][nx]
  T* vt;          // [4][nc] limited moments (the state's v, w keep the unlimited ones)
  T* wt;
  // the state as the limiter and the face kernels read it, in the compute type: for double the
  // state array and prim (set by the launcher); for float copies written by the kernels that
  // produce the state, so each cell is converted once per stage, not once per stencil use
  T* qt;          // [4][nc]
  T* primt;       // [4][nc] u, v, h, sqrt|rho|
};

template <typename T>
size_t work_bytes_h(int nx, int ny) {
  const size_t nc = size_t(nx) * ny, nxf = size_t(nx + 1) * ny, nyf = size_t(ny + 1) * nx;
  return 16 * nc * sizeof(T) + (24 + 7 + 12) * (nxf + nyf) * sizeof(T) + 256 * 12;
}

template <typename T>
WorkH<T> carve_h(void* base, int nx, int ny) {
  const size_t nc = size_t(nx) * ny, nxf = size_t(nx + 1) * ny, nyf = size_t(ny + 1) * nx;
  char* p = static_cast<char*>(base);
  auto take = [&](size_t bytes) {
    char* r = p;
    p += (bytes + 255) & ~size_t(255);
    return r;
  };
  WorkH<T> w;
  w.xc = reinterpret_cast<T*>(take(24 * nxf * sizeof(T)));
  w.xroe = reinterpret_cast<T*>(take(7 * nxf * sizeof(T)));
  w.yc = reinterpret_cast<T*>(take(24 * nyf * sizeof(T)));
  w.yroe = reinterpret_cast<T*>(take(7 * nyf * sizeof(T)));
  w.fx = reinterpret_cast<T*>(take(12 * nxf * sizeof(T)));
  w.fy = reinterpret_cast<T*>(take(12 * nyf * sizeof(T)));
  w.vt = reinterpret_cast<T*>(take(4 * nc * sizeof(T)));
  w.wt = reinterpret_cast<T*>(take(4 * nc * sizeof(T)));
  w.prim = nullptr;
  w.qt = w.primt = nullptr;
  T* prim = reinterpret_cast<T*>(take(4 * nc * sizeof(T)));
  if constexpr (std::is_same<T, double>::value) {
    w.prim = prim;
  } else {
    w.primt = prim;
    w.qt = reinterpret_cast<T*>(take(4 * nc * sizeof(T)));
  }
  return w;
}

int hermite2d_fp64_setup(hteno_solver* s);
void hermite2d_fp64_step(hteno_solver* s, const GeoH& G);
void hermite2d_fp64_prim(hteno_solver* s, const GeoH& G);

namespace {

__constant__ DevConst c_dev;
__device__ DevConst g_dev;  // the same in global memory (double: par::ldk)
unsigned long long g_mask = 0;
std::mutex g_mu;

#include "common_kernels.cuh"

__device__ __forceinline__ void cell_prim(double g1, const double* q, double& u, double& v,
                                          double& p, double& h, double& sr) {
  u = q[1] / q[0];
  v = q[2] / q[0];
  p = (q[3] - 0.5 * (q[1] * u + q[2] * v)) * g1;
  h = (q[3] + p) / q[0];
  sr = sqrt(fabs(q[0]));
}
__device__ __forceinline__ double cell_max_speed(double gamma, double rho, double u, double v,
                                                 double p) {
  const double c = sqrt(fabs(gamma * p / rho));
  return fmax(fmax(u - c, fabs(u + c)), fmax(v - c, fabs(v + c)));
}

__global__ void kh_prim(GeoH G, const double* __restrict__ q, double* __restrict__ prim,
                        StepState* st, int do_max) {
  const size_t nc = size_t(G.nx) * G.ny;
  const size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
  double ms = 0.0;
  if (k < nc) {
    double qq[4] = {q[k], q[nc + k], q[2 * nc + k], q[3 * nc + k]};
    double u, v, p, h, sr;
    cell_prim(G.g1, qq, u, v, p, h, sr);
    prim[k] = u;
    prim[nc + k] = v;
    prim[2 * nc + k] = h;
    prim[3 * nc + k] = sr;
    ms = cell_max_speed(G.gamma, qq[0], u, v, p);
  }
  if (do_max) block_max_to(ms, &st->maxbits);
}

// Mixed precision, after a new state: the float copies of the state and of its primitives that
// the face kernels read, and the first dt's max wave speed.  The primitives are those of cell_prim
// rounded to float.  Bound by the FP64 pipe: the divisions and square roots took 0.71 ms at 2048^2.
// So they are first computed from refined float reciprocals and roots (14 FP64 operations, relative
// errors below 2^-41), which round to the same floats unless a value lies that close to the middle of
// two of them; there, in odd ranges and for the speed (SpeedFilter) cell_prim decides.  Now 0.25 ms.
// Small grids take cell_prim in every cell (speed_rule.h).
__device__ __forceinline__ bool float_sure(double x) {
  const unsigned lo = unsigned(__double2loint(x)) & 0x1fffffffu;  // the bits a float drops
  const int e = ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
  return (lo - (0x10000000u - 16384u) > 32768u && e > -100 && e < 100) || x == 0.0;
}
__global__ void kh_prim_f(GeoH G, const double* __restrict__ q, float* __restrict__ qt,
                          float* __restrict__ primt, StepState* st, bool filter) {
  __shared__ unsigned found;
  const size_t nc = size_t(G.nx) * G.ny;
  if (!filter) {  // a cell a thread
    const size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
    double m = 0.0;
    if (k < nc) {
      const double qq[4] = {q[k], q[nc + k], q[2 * nc + k], q[3 * nc + k]};
      double u, v, p, h, sr;
      cell_prim(G.g1, qq, u, v, p, h, sr);
#pragma unroll
      for (int e = 0; e < 4; ++e) qt[e * nc + k] = mix::d2f(qq[e]);
      primt[k] = mix::d2f(u);
      primt[nc + k] = mix::d2f(v);
      primt[2 * nc + k] = mix::d2f(h);
      primt[3 * nc + k] = mix::d2f(sr);
      m = cell_max_speed(G.gamma, qq[0], u, v, p);
    }
    block_max_to(m, &st->maxbits);
    return;
  }
  mix::SpeedFilter F(&found, &st->maxbits, G.g1, G.gamma, nc);
  const float g1f = 1.0f + fabsf(float(G.g1));
  double ms = 0.0;
  for (size_t k = F.k; k < F.end; k += blockDim.x) {
    double qq[4] = {q[k], q[nc + k], q[2 * nc + k], q[3 * nc + k]};
    float f[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) qt[e * nc + k] = f[e] = mix::d2f(qq[e]);
    double ir = mix::f2d(__frcp_rn(f[0]));
    ir = fma(ir, fma(-qq[0], ir, 1.0), ir);
    const double s0 = mix::f2d(sqrtf(f[0]));
    double u = qq[1] * ir, v = qq[2] * ir;
    const double ke2 = fma(qq[1], u, qq[2] * v);
    double p = fma(-0.5, ke2, qq[3]) * G.g1;
    const double hr = qq[3] + p;
    double h = hr * ir, sr = fma(fma(-s0, s0, qq[0]), mix::f2d(0.5f * __frcp_rn(sqrtf(f[0]))), s0);
    const float big = (fabsf(f[3]) + mix::d2f(ke2)) * g1f;
    const bool sure = f[0] > 1e-18f && f[0] < 1e18f && float_sure(u) && float_sure(v) && float_sure(h) && float_sure(sr) &&
                      (u != 0.0 || qq[1] == 0.0) && (v != 0.0 || qq[2] == 0.0) && big < 1e30f &&
                      fabsf(mix::d2f(hr)) * 16.0f >= big;
    const bool fast = F.may_exceed(qq);
    if (!sure || fast) {
      cell_prim(G.g1, qq, u, v, p, h, sr);
      const double m = cell_max_speed(G.gamma, qq[0], u, v, p);
      ms = fmax(ms, m);
      F.add(qq, m);
    }
    primt[k] = mix::d2f(u);
    primt[nc + k] = mix::d2f(v);
    primt[2 * nc + k] = mix::d2f(h);
    primt[3 * nc + k] = mix::d2f(sr);
  }
  block_max_to(ms, &st->maxbits);
}

// ---- the limiter ---------------------------------------------------------------------------------
// The reference's limiter is a Gauss-Seidel sweep along every line (row j of field e walking i on
// v, column i walking j on w): each cell reads its left neighbour's limited value, so a line is one
// serial chain, ~110 FP64 operations (64 cycles each) or ~70 dependent float operations per cell.
// The chain forgets quickly (a cell passes on about a quarter of its left neighbour's change), so
// a line is cut into segments that sweep side by side: every segment first starts from a guess of its
// left neighbour's value (the unlimited moment; in double the float sweep of the kLimWarm cells before
// it, which costs next to nothing beside one cell in double); then, as long as a segment's left
// neighbour came out with other bits than it was computed from, it sweeps again from its first cell
// and stops at the first cell whose bits do not change.  When nothing changes any more every cell
// has been computed from its final left neighbour: the bits of the one sweep, whatever the data.
// (Segment k is final after k such passes at the latest.  Bits usually agree again after about 15
// cells in double, 28 without the float guess, and 12-21 in float; a tail that vanishes into constant
// data takes longer, in double on the short form at_flat.)
//
// Threads of a block: `lines` lines (16 or 32, the fast index) x segments.  Blocks [0, nbx): x
// lines; [nbx, ...): y lines.  The neighbour beyond the last cell is the zero-gradient ghost, the
// one before the first cell is the first cell (unlimited values).  Limited moments go to vt, wt:
// the unlimited ones stay where the later stages of a step read them.  A y line's cells are read
// across the lanes (coalesced); in float an x line's come through shared memory in chunks of kLimC
// cells of the warp's 32 lines, loaded and stored along the rows (kStaged; in double the arithmetic
// hides the scattered loads).
constexpr int kLimC = 16, kLimWarm = 24;

template <typename T, bool kStaged>
__global__ void __launch_bounds__(256) kh_limit(GeoH G, HermiteK<T> K, const T* __restrict__ q,
                                                const double* __restrict__ v, const double* __restrict__ w,
                                                T* __restrict__ vt, T* __restrict__ wt, int lines, int segx, int segy,
                                                int nbx, const StepState* st) {
  if (st->done) return;
  __shared__ T last[256];  // the limited value of each segment's last cell
  const bool xd = int(blockIdx.x) < nbx;
  const int b = xd ? int(blockIdx.x) : int(blockIdx.x) - nbx;
  const int nl = xd ? G.ny : G.nx;  // number of lines
  const int n = xd ? G.nx : G.ny;   // length of a line
  const int nlb = (nl + lines - 1) / lines;
  const int e = b / nlb, seg = threadIdx.x / lines, segs = xd ? segx : segy;
  const int l0 = (b - e * nlb) * lines, line = l0 + int(threadIdx.x) - seg * lines;
  const int len = (n + segs - 1) / segs, c0 = min(n, seg * len), c1 = min(n, c0 + len);
  const bool live = line < nl && c0 < c1;  // (no thread of a segment past the direction's number)
  const size_t field = size_t(e) * G.nx * G.ny;
  const size_t base = field + (xd ? size_t(line) * G.nx : size_t(line));
  const size_t step = xd ? 1 : size_t(G.nx);
  const double* __restrict__ d = xd ? v : w;
  T* __restrict__ out = xd ? vt : wt;
  T used = T(0);  // the left neighbour's value the segment was computed from
  // cells c0 .. of the segment from the left value dl; with `again` up to the first unchanged cell
  auto sweep = [&](T dl, bool again) {
    LimitSweep<T> s(K, q[base + size_t(max(c0 - 1, 0)) * step], q[base + size_t(c0) * step]);
    size_t k = base + size_t(c0) * step, kr = base + size_t(min(c0 + 1, n - 1)) * step;
    T ur = q[kr], dr = from_d<T>(d[kr]);
    for (int i = c0; i < c1; ++i, k += step) {
      s.next(ur, dr);
      if (i + 1 < c1) {  // in flight during this cell's arithmetic
        kr = base + size_t(min(i + 2, n - 1)) * step;
        ur = q[kr];
        dr = from_d<T>(d[kr]);
      }
      if constexpr (std::is_same<T, double>::value) dl = again && s.flat() ? s.at_flat(dl) : s.at(dl);
      else dl = s.at(dl);
      if (again && same_bits(dl, out[k])) return;
      out[k] = dl;
    }
    last[threadIdx.x] = dl;
  };
  if (live) used = from_d<T>(d[base + size_t(max(c0 - 1, 0)) * step]);
  if constexpr (std::is_same<T, double>::value) {
    if (live && c0 > kLimWarm) {
      auto uf = [&](int i) { return mix::d2f(q[base + size_t(i) * step]); };
      auto df = [&](int i) { return mix::d2f(d[base + size_t(i) * step]); };
      LimitSweep<float> s(K, uf(c0 - kLimWarm - 1), uf(c0 - kLimWarm));
      float x = df(c0 - kLimWarm - 1);
      for (int i = c0 - kLimWarm; i < c0; ++i) {  // the limited value of cell i
        s.next(uf(i + 1), df(i + 1));
        x = s.at(x);
      }
      if (fabsf(x) <= 3.4e38f) used = mix::f2d(x);
    }
  }
  if constexpr (kStaged) {
    __shared__ T su[8][kLimC][33], sd[8][kLimC][33];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;  // a warp: 32 lines, one segment
    if (xd && c0 < c1) {
      const size_t mine = field + size_t(min(line, nl - 1)) * G.nx;
      LimitSweep<T> s(K, q[mine + max(c0 - 1, 0)], q[mine + c0]);
      T dl = used;
      for (int a = c0; a < c1; a += kLimC) {
        const int cnt = min(kLimC, c1 - a);
        __syncwarp();
#pragma unroll 4
        for (int j = 0; j < 32 * kLimC / 32; ++j) {  // the right neighbours of cells a .. a + 15
          const int r = j * (32 / kLimC) + lane / kLimC, c = lane % kLimC;
          const size_t kr = field + size_t(min(l0 + r, nl - 1)) * G.nx + min(a + c + 1, n - 1);
          su[wid][c][r] = q[kr];
          sd[wid][c][r] = from_d<T>(d[kr]);
        }
        __syncwarp();
        for (int c = 0; c < cnt; ++c) {
          s.next(su[wid][c][lane], sd[wid][c][lane]);
          dl = s.at(dl);
          sd[wid][c][lane] = dl;
        }
        __syncwarp();
#pragma unroll 4
        for (int j = 0; j < 32 * kLimC / 32; ++j) {
          const int r = j * (32 / kLimC) + lane / kLimC, c = lane % kLimC;
          if (l0 + r < nl && c < cnt) out[field + size_t(l0 + r) * G.nx + a + c] = sd[wid][c][r];
        }
      }
      last[threadIdx.x] = dl;
    } else if (live) {
      sweep(used, false);
    }
  } else if (live) {
    sweep(used, false);
  }
  for (int pass = 1; pass < segs; ++pass) {
    __syncthreads();
    const T left = live && seg ? last[threadIdx.x - lines] : used;
    const bool redo = live && !same_bits(left, used);
    if (!__syncthreads_or(redo)) break;
    if (redo) {
      used = left;
      sweep(left, true);
    }
  }
}

// Characteristic reconstruction of every face: HTENO of value and derivative from u and the moment along
// the sweep, TENO5 of the cross moment.  In float bound by instruction issue (67 % of the slots; FMA pipe
// 62 %, ALU 46 %): projections of two cells and both sides of a reconstruction in packed pairs, the
// weights per cut-off pattern in shared memory.  2048^2: 440 -> 405 us, the same bits.
template <typename T, int DIR>
__global__ void __launch_bounds__(kHFaceThreads, kHFaceBlocks<T>) kh_faces(GeoH G, HermiteK<T> K,
                                                         const T* __restrict__ q,
                                                         const T* __restrict__ v,
                                                         const T* __restrict__ w,
                                                         const T* __restrict__ prim,
                                                         T* __restrict__ fc, T* __restrict__ froe,
                                                         const StepState* st) {
  if (st && st->done) return;
  __shared__ typename std::conditional<std::is_same<T, double>::value, char, HermiteTab>::type tab;
  __shared__ typename std::conditional<std::is_same<T, double>::value, char[28][1], f2[28][kHFaceThreads]>::type cv;
  if constexpr (!std::is_same<T, double>::value) load_hermite_tab(tab, K, c_dev);
  const int nf = DIR == 1 ? G.nx + 1 : G.ny + 1;
  const int nt = DIR == 1 ? G.ny : G.nx;
  const long idx = blockIdx.x * long(blockDim.x) + threadIdx.x;
  if (idx >= long(nf) * nt) return;
  int f, t;
  if (DIR == 1) { f = int(idx % nf); t = int(idx / nf); }
  else { t = int(idx % nt); f = int(idx / nt); }
  const size_t nc = size_t(G.nx) * G.ny;
  const int ns = DIR == 1 ? G.nx : G.ny;
  auto cell = [&](int s) -> size_t {
    const int m = bmap(s, ns, HTENO_BC_ZEROGRAD);
    return DIR == 1 ? size_t(t) * G.nx + m : size_t(m) * G.nx + t;
  };
  const T* mn = DIR == 1 ? v : w;  // moment along the sweep (HTENO)
  const T* mt = DIR == 1 ? w : v;  // cross moment (TENO5)
  const size_t ca = cell(f - 1), cb = cell(f);
  const size_t nface = size_t(nf) * nt;
  const size_t o = DIR == 1 ? size_t(t) * nf + f : size_t(f) * nt + t;
  if constexpr (std::is_same<T, double>::value) {
    const par::Eig E = par::eig(G.g1, DIR, prim[3 * nc + ca], prim[ca], prim[nc + ca],
                                prim[2 * nc + ca], prim[3 * nc + cb], prim[cb], prim[nc + cb],
                                prim[2 * nc + cb]);
    {
      double A[4][4], B[4][4];
      for (int m = 0; m < 4; ++m) {
        const size_t c = cell(f - 2 + m);
        const double a4[4] = {q[c], q[nc + c], q[2 * nc + c], q[3 * nc + c]};
        const double b4[4] = {mn[c], mn[nc + c], mn[2 * nc + c], mn[3 * nc + c]};
        double ca4[4], cb4[4];
        par::left(E, DIR, a4, ca4);
        par::left(E, DIR, b4, cb4);
        for (int r = 0; r < 4; ++r) {
          A[r][m] = ca4[r];
          B[r][m] = cb4[r];
        }
      }
      for (int r = 0; r < 4; ++r) {
        double h[4];
        par::hermite_recon(g_dev, K, 0, A[r], B[r], h);
        for (int a = 0; a < 4; ++a) fc[(a * 4 + r) * nface + o] = h[a];
      }
    }
    {
      double C[4][6];
      for (int m = 0; m < 6; ++m) {
        const size_t c = cell(f - 3 + m);
        const double c4[4] = {mt[c], mt[nc + c], mt[2 * nc + c], mt[3 * nc + c]};
        double cc[4];
        par::left(E, DIR, c4, cc);
        for (int r = 0; r < 4; ++r) C[r][m] = cc[r];
      }
      for (int r = 0; r < 4; ++r) {
        double a, b;
        par::lagrange_recon(g_dev, HTENO_RECON_TENO5, C[r], a, b);
        fc[(4 * 4 + r) * nface + o] = a;
        fc[(5 * 4 + r) * nface + o] = b;
      }
    }
    par::eig_store(E, froe + o, nface);
  } else {
    const Roe2<T> R = roe2<T>(T(G.g1), prim[3 * nc + ca], prim[ca], prim[nc + ca], prim[2 * nc + ca],
                              prim[3 * nc + cb], prim[cb], prim[nc + cb], prim[2 * nc + cb]);
    const LeftRows L = left_rows(R, DIR);
    // characteristic values of cells f + c0, f + c0 + 1 (pairs) of the conserved fields x
    auto project = [&](const T* x, int c0, f2* c) {
      const size_t a = cell(f + c0), b = cell(f + c0 + 1);
      const f2 w[4] = {pack(x[a], x[b]), pack(x[nc + a], x[nc + b]), pack(x[2 * nc + a], x[2 * nc + b]),
                       pack(x[3 * nc + a], x[3 * nc + b])};
      project2(L, DIR, w, c);
    };
    // the pairs wait in shared memory (per thread), one field's at a time in registers
    auto put = [&](int k, const T* x, int c0) {
      f2 c[4];
      project(x, c0, c);
#pragma unroll
      for (int r = 0; r < 4; ++r) cv[4 * k + r][threadIdx.x] = c[r];
    };
    put(0, q, -2);
    put(1, q, 0);
    put(2, mn, -2);
    put(3, mn, 0);
    put(4, mt, -3);
    put(5, mt, -1);
    put(6, mt, 1);
#pragma unroll 1
    for (int r = 0; r < 4; ++r) {
      auto get = [&](int k) { return cv[4 * k + r][threadIdx.x]; };
      const HtenoSides h = hteno_sides(tab, K.dif, get(0), get(1), get(2), get(3));
      fc[(0 * 4 + r) * nface + o] = lo(h.u);
      fc[(1 * 4 + r) * nface + o] = hi(h.u);
      fc[(2 * 4 + r) * nface + o] = lo(h.d);
      fc[(3 * 4 + r) * nface + o] = hi(h.d);
      const f2 u = teno5_sides(c_dev, tab, get(4), get(5), get(6));
      fc[(4 * 4 + r) * nface + o] = lo(u);
      fc[(5 * 4 + r) * nface + o] = hi(u);
    }
    froe[0 * nface + o] = R.vxm;
    froe[1 * nface + o] = R.vym;
    froe[2 * nface + o] = R.hm;
    froe[3 * nface + o] = R.qm;
    froe[4 * nface + o] = R.cm;
    froe[5 * nface + o] = R.rcm;
    froe[6 * nface + o] = R.b1;
  }
}

template <typename T, int DIR>
__global__ void __launch_bounds__(kHFluxThreads) kh_flux(GeoH G, const T* __restrict__ fc,
                                                        const T* __restrict__ froe,
                                                        T* __restrict__ F, const StepState* st) {
  // In float bound by instruction issue (66 % of the slots, 4600 per warp of which GL3 half): GL3 and the
  // back-projection take both sides of a face in packed pairs (2048^2: 700 -> 518 us, the same bits).
  // GL3 values of the 24 face arrays at the 3 Gauss points, per thread, in shared memory: for
  // float the (minus, plus) pairs as [pair][point][thread] (a warp's accesses fall in distinct banks);
  // for double [thread][array][point] with a one-value pad per thread (par::gl3 writes 3 contiguous
  // values; the odd stride of 73 values spreads a warp's 8-byte accesses over all banks)
  typedef typename std::conditional<std::is_same<T, double>::value, double, f2>::type Sg;
  constexpr int kSgT = std::is_same<T, double>::value ? 73 : 36;
  __shared__ Sg sg[kHFluxThreads * kSgT];
  auto gat = [&](int a, int m) -> Sg& {
    if constexpr (std::is_same<T, double>::value) return sg[threadIdx.x * kSgT + a * 3 + m];
    else return sg[(a * 3 + m) * kHFluxThreads + threadIdx.x];
  };
  if (st && st->done) return;
  const int nf = DIR == 1 ? G.nx + 1 : G.ny + 1;
  const int nt = DIR == 1 ? G.ny : G.nx;
  const long idx = blockIdx.x * long(blockDim.x) + threadIdx.x;
  const bool live = idx < long(nf) * nt;
  int f = 0, t = 0;
  if (live) {
    if (DIR == 1) { f = int(idx % nf); t = int(idx / nf); }
    else { t = int(idx % nt); f = int(idx / nt); }
  }
  const size_t nface = size_t(nf) * nt;
  auto fidx = [&](int tt) -> size_t {
    const int m = bmap(tt, nt, HTENO_BC_ZEROGRAD);
    return DIR == 1 ? size_t(m) * nf + f : size_t(f) * nt + m;
  };
  if (!live) return;
  size_t nb[5];
#pragma unroll
  for (int m = 0; m < 5; ++m) nb[m] = fidx(t - 2 + m);
  if constexpr (std::is_same<T, double>::value) {
    for (int a = 0; a < 24; ++a) {
      T u5[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) u5[m] = fc[size_t(a) * nface + nb[m]];
      par::gl3(g_dev, u5, &gat(a, 0));
    }
  } else {
    // pair a: field a % 4 of kind a / 4 (u, normal and tangential derivative), both sides of the face
    for (int a = 0; a < 12; ++a) {
      const T* fa = fc + size_t(8 * (a / 4) + a % 4) * nface;
      f2 u5[5];
#pragma unroll
      for (int m = 0; m < 5; ++m) u5[m] = pack(fa[nb[m]], fa[4 * nface + nb[m]]);
      const Gl3f g = gl3_pair<true>(c_dev, u5[0], u5[1], u5[2], u5[3], u5[4]);
      gat(a, 0) = g.a;
      gat(a, 1) = g.b;
      gat(a, 2) = g.c;
    }
  }
  const size_t o = nb[2];
  T acc[12];
  if constexpr (std::is_same<T, double>::value) {
    const par::Eig E = par::eig_load(DIR, froe + o, nface);
    par::fp Fk[12];
    for (int m = 0; m < 3; ++m) {
      par::fp X[6][4];
      for (int a = 0; a < 6; ++a) {
        const par::fp c[4] = {gat(4 * a + 0, m), gat(4 * a + 1, m), gat(4 * a + 2, m), gat(4 * a + 3, m)};
        par::right(E, DIR, c, X[a]);
      }
      par::fp fu[4], fn[4], ft[4];
      const par::Sides S = par::sides_of(G.gamma, G.g1, DIR, X[0], X[1]);
      par::rusanov(DIR, E, S, X[0], X[1], fu);
      par::drusanov(G.gamma, G.g1, G.g3, DIR, E, S, X[0], X[1], X[2], X[3], fn);
      par::drusanov(G.gamma, G.g1, G.g3, DIR, E, S, X[0], X[1], X[4], X[5], ft);
      const par::fp wm = par::ldk(g_dev.gl3w[m]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        Fk[k] = m == 0 ? wm * fu[k] : Fk[k] + wm * fu[k];
        Fk[4 + k] = m == 0 ? wm * fn[k] : Fk[4 + k] + wm * fn[k];
        Fk[8 + k] = m == 0 ? wm * ft[k] : Fk[8 + k] + wm * ft[k];
      }
    }
#pragma unroll
    for (int k = 0; k < 12; ++k) acc[k] = Fk[k].v;
  } else {
    Roe2<T> R;
    R.vxm = froe[o];
    R.vym = froe[nface + o];
    R.hm = froe[2 * nface + o];
    R.qm = froe[3 * nface + o];
    R.cm = froe[4 * nface + o];
    R.rcm = froe[5 * nface + o];
    R.b1 = froe[6 * nface + o];
    const T gm = T(G.gamma), g1 = T(G.g1);
    for (int m = 0; m < 3; ++m) {
      T X[6][4];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const f2 c[4] = {gat(4 * a + 0, m), gat(4 * a + 1, m), gat(4 * a + 2, m), gat(4 * a + 3, m)};
        f2 x[4];
        right2(R, DIR, c, x);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          X[2 * a][k] = lo(x[k]);
          X[2 * a + 1][k] = hi(x[k]);
        }
      }
      T fu[4], fn[4], ft[4];
      rusanov2(gm, g1, DIR, R, X[0], X[1], fu);
      drusanov2(gm, g1, DIR, R, X[0], X[1], X[2], X[3], fn);
      drusanov2(gm, g1, DIR, R, X[0], X[1], X[4], X[5], ft);
      const T wm = Cst<T>::gl3w(c_dev, m);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        acc[k] = m == 0 ? wm * fu[k] : acc[k] + wm * fu[k];
        acc[4 + k] = m == 0 ? wm * fn[k] : acc[4 + k] + wm * fn[k];
        acc[8 + k] = m == 0 ? wm * ft[k] : acc[8 + k] + wm * ft[k];
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 12; ++k) F[size_t(k) * nface + o] = acc[k];
}

// rhs (:710-730) and RungeKutta3 (:733-782) for u, v, w: stage 1 starts from the limited moments
// (vt, wt) and saves them, the later stages combine with the unlimited stage values in v, w.
template <typename T>
__global__ void __launch_bounds__(256, 4) kh_update(GeoH G, int stage, const T* __restrict__ fx, const T* __restrict__ fy,
                          double* __restrict__ q, double* __restrict__ q0,
                          double* __restrict__ v, double* __restrict__ v0,
                          const T* __restrict__ vt, double* __restrict__ w,
                          double* __restrict__ w0, const T* __restrict__ wt,
                          double* __restrict__ prim, float* __restrict__ qt,
                          float* __restrict__ primt, StepState* st) {
  if (st->done) return;
  const size_t nc = size_t(G.nx) * G.ny;
  const size_t k = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
  double ms = 0.0;
  int bad = 0;
  if (k < nc) {
    const int i = int(k % G.nx), j = int(k / G.nx);
    const size_t nxf = size_t(G.nx + 1) * G.ny, nyf = size_t(G.ny + 1) * G.nx;
    const size_t ox = size_t(j) * (G.nx + 1) + i, oy = size_t(j) * G.nx + i;
    const double dt = st->dt;
    double qn[4];
    if constexpr (std::is_same<T, float>::value) {
      // mixed precision: the residual from the float fluxes in float (a difference of two
      // nearby fluxes is exact in float; otherwise its rounding is far below the fluxes' own),
      // the RK stage in double with FMAs; the conversions on the integer pipes; primitives with
      // a refined float reciprocal of rho.  The FP64 pipe (1/64 of the float rate) does only
      // the accumulation and the primitives, its factors in vector registers and the tests on the
      // bits (2048^2: 580 -> 519 us a stage).
      auto rhs = [&](int kx, int ky, int e) {
        const float dfx = fx[(kx + e) * nxf + ox] - fx[(kx + e) * nxf + ox + 1];
        const float dfy = fy[(ky + e) * nyf + oy] - fy[(ky + e) * nyf + oy + G.nx];
        return mix::f2d(fmaf(dfx, G.rdxf, dfy * G.rdyf));
      };
      const mix::RkStage rk = mix::rk_stage(stage, dt);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const double ru = rhs(0, 0, e), rv = rhs(4, 8, e), rw = rhs(8, 4, e);
        const size_t c = size_t(e) * nc + k;
        double bq, bv, bw, cq = q[c], cv, cw;
        if (stage == 1) {
          bq = cq; bv = to_d<T>(vt[c]); bw = to_d<T>(wt[c]);
          q0[c] = bq; v0[c] = bv; w0[c] = bw;
          cv = bv; cw = bw;
        } else {
          bq = q0[c]; bv = v0[c]; bw = w0[c];
          cv = v[c]; cw = w[c];
        }
        qn[e] = rk(bq, cq, ru);
        const double nv = rk(bv, cv, rv);
        const double nw = rk(bw, cw, rw);
        q[c] = qn[e];
        qt[c] = mix::d2f(qn[e]);
        v[c] = nv;
        w[c] = nw;
      }
      const float fr = mix::d2f(qn[0]);
      double ir = mix::f2d(__frcp_rn(fr));
      ir = fma(ir, fma(-qn[0], ir, 1.0), ir);
      const double u = qn[1] * ir, vv = qn[2] * ir;
      const double p = (qn[3] - 0.5 * (qn[1] * u + qn[2] * vv)) * G.g1;
      primt[k] = mix::d2f(u);
      primt[nc + k] = mix::d2f(vv);
      primt[2 * nc + k] = mix::d2f((qn[3] + p) * ir);
      primt[3 * nc + k] = Cst<float>::sqrt_(fabsf(fr));
      if (stage == 3) {
        const float fu = mix::d2f(u), fv = mix::d2f(vv);
        const float cs = sqrtf(fabsf(float(G.gamma) * mix::d2f(p) / fr));
        ms = mix::f2d(fmaxf(fmaxf(fu - cs, fabsf(fu + cs)), fmaxf(fv - cs, fabsf(fv + cs))));
      }
      bad = (par::nan_bits(qn[0]) || par::nan_bits(qn[1]) || par::nan_bits(qn[2]) || par::nan_bits(qn[3]) ||
             par::nan_bits(p)) ? 1 : 0;
      bad |= (par::nonpositive_bits(qn[0]) || par::nonpositive_bits(p)) ? 2 : 0;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // kinds: x-sweep (0 u, 1 v, 2 w), y-sweep (0 u, 1 w, 2 v)
        const double ru = ((double(fx[(0 + e) * nxf + ox]) - double(fx[(0 + e) * nxf + ox + 1])) * G.dy +
                           (double(fy[(0 + e) * nyf + oy]) - double(fy[(0 + e) * nyf + oy + G.nx])) * G.dx) / G.area + 0.0;
        const double rv = ((double(fx[(4 + e) * nxf + ox]) - double(fx[(4 + e) * nxf + ox + 1])) * G.dy +
                           (double(fy[(8 + e) * nyf + oy]) - double(fy[(8 + e) * nyf + oy + G.nx])) * G.dx) / G.area + 0.0;
        const double rw = ((double(fx[(8 + e) * nxf + ox]) - double(fx[(8 + e) * nxf + ox + 1])) * G.dy +
                           (double(fy[(4 + e) * nyf + oy]) - double(fy[(4 + e) * nyf + oy + G.nx])) * G.dx) / G.area + 0.0;
        const size_t c = size_t(e) * nc + k;
        double bq, bv, bw, cq = q[c], cv, cw;
        if (stage == 1) {
          bq = cq; bv = vt[c]; bw = wt[c];  // save() after the first rhs: limited moments
          q0[c] = bq; v0[c] = bv; w0[c] = bw;
          cv = bv; cw = bw;
        } else {
          bq = q0[c]; bv = v0[c]; bw = w0[c];
          cv = v[c]; cw = w[c];            // unlimited stage values (cell.v1 / cell.v2)
        }
        qn[e] = par::rk3(bq, cq, ru, dt, stage);
        const double nv = par::rk3(bv, cv, rv, dt, stage);
        const double nw = par::rk3(bw, cw, rw, dt, stage);
        q[c] = qn[e];
        v[c] = nv;
        w[c] = nw;
      }
      double u, vv, p, h, sr;
      cell_prim(G.g1, qn, u, vv, p, h, sr);
      prim[k] = u;
      prim[nc + k] = vv;
      prim[2 * nc + k] = h;
      prim[3 * nc + k] = sr;
      if (stage == 3) ms = cell_max_speed(G.gamma, qn[0], u, vv, p);
      bad = (isnan(qn[0]) || isnan(qn[1]) || isnan(qn[2]) || isnan(qn[3])) ? 1 : 0;
      bad |= (qn[0] <= 0.0 || p <= 0.0) ? 2 : 0;
    }
  }
  if (stage == 3) block_max_to(ms, &st->maxbits);
  if (bad) atomicOr(&st->status, bad);
}

GeoH geo_of(const hteno_solver* s) {
  GeoH G;
  G.nx = s->cfg.nx;
  G.ny = s->cfg.ny;
  G.dx = s->dx;
  G.dy = s->dy;
  G.area = s->dx * s->dy;
  G.gamma = s->cfg.gamma;
  G.g1 = s->cfg.gamma - 1.0;
  G.g3 = s->cfg.gamma - 3.0;
  G.rdx = 1.0 / s->dx;
  G.rdy = 1.0 / s->dy;
  G.rdxf = float(G.rdx);
  G.rdyf = float(G.rdy);
  return G;
}

// The limiter's launch (limit_rule.h).
template <typename T>
void launch_limit(hteno_solver* s, const GeoH& G, const HermiteK<T>& K, const WorkH<T>& W) {
  const LimitShape L = limit_shape(G.nx, G.ny);
  const int nbx = 4 * ((G.ny + L.lines - 1) / L.lines), nby = 4 * ((G.nx + L.lines - 1) / L.lines);
  const unsigned threads = unsigned(L.lines * std::max(L.segx, L.segy));  // whole warps
  constexpr bool staged = std::is_same<T, float>::value;
  if (L.wide && staged)
    kh_limit<T, staged><<<unsigned(nbx + nby), threads, 0, s->stream>>>(G, K, W.qt, s->v, s->w, W.vt, W.wt, L.lines,
                                                                       L.segx, L.segy, nbx, s->dstate);
  else
    kh_limit<T, false><<<unsigned(nbx + nby), threads, 0, s->stream>>>(G, K, W.qt, s->v, s->w, W.vt, W.wt, L.lines,
                                                                      L.segx, L.segy, nbx, s->dstate);
}

template <typename T>
void launch_step(hteno_solver* s, const GeoH& G) {
  cudaStream_t cs = s->stream;
  WorkH<T> W = carve_h<T>(s->work, G.nx, G.ny);
  if constexpr (std::is_same<T, double>::value) {
    W.qt = s->q;
    W.primt = W.prim;
  }
  const HermiteK<T> K = make_hermite_k<T>(s->dx);  // setGridSize(dx) for both directions
  const int nx = G.nx, ny = G.ny;
  const long nxf = long(nx + 1) * ny, nyf = long(ny + 1) * nx;
  const size_t nc = size_t(nx) * ny;
  const double ncd = double(nc);
  const int k_l = trace_kind(s, "h_limit", ncd * 4 * 8 * 6, 0);
  const int k_fx = trace_kind(s, "h_faces_x", ncd * 128 + double(nxf) * 31 * sizeof(T), 0);
  const int k_fy = trace_kind(s, "h_faces_y", ncd * 128 + double(nyf) * 31 * sizeof(T), 0);
  const int k_x = trace_kind(s, "h_flux_x", double(nxf) * 43 * sizeof(T), 0);
  const int k_y = trace_kind(s, "h_flux_y", double(nyf) * 43 * sizeof(T), 0);
  const int k_u = trace_kind(s, "h_update", ncd * 8 * 40 + double(nxf + nyf) * 12 * sizeof(T), 0);
  k_begin_step<<<1, 1, 0, cs>>>(s->dstate);
  for (int stage = 1; stage <= 3; ++stage) {
    trace_begin(s, k_l);
    launch_limit<T>(s, G, K, W);
    trace_end(s);
    // the y faces and fluxes beside the x ones on the side stream (one stream while timing)
    // (if the fork cannot be recorded, the y kernels stay on the solver's stream)
    const bool fork = s->side_stream && !s->timing &&
                      cudaEventRecord(s->fork_ev, cs) == cudaSuccess &&
                      cudaStreamWaitEvent(s->side_stream, s->fork_ev, 0) == cudaSuccess;
    cudaStream_t ys = fork ? s->side_stream : cs;
    trace_begin(s, k_fx);
    kh_faces<T, 1><<<unsigned((nxf + kHFaceThreads - 1) / kHFaceThreads), kHFaceThreads, 0, cs>>>(
        G, K, W.qt, W.vt, W.wt, W.primt, W.xc, W.xroe, s->dstate);
    trace_end(s);
    trace_begin(s, k_fy);
    kh_faces<T, 2><<<unsigned((nyf + kHFaceThreads - 1) / kHFaceThreads), kHFaceThreads, 0, ys>>>(
        G, K, W.qt, W.vt, W.wt, W.primt, W.yc, W.yroe, s->dstate);
    trace_end(s);
    trace_begin(s, k_x);
    kh_flux<T, 1><<<unsigned((nxf + kHFluxThreads - 1) / kHFluxThreads), kHFluxThreads, 0, cs>>>(
        G, W.xc, W.xroe, W.fx, s->dstate);
    trace_end(s);
    trace_begin(s, k_y);
    kh_flux<T, 2><<<unsigned((nyf + kHFluxThreads - 1) / kHFluxThreads), kHFluxThreads, 0, ys>>>(
        G, W.yc, W.yroe, W.fy, s->dstate);
    trace_end(s);
    // the join; if it cannot be recorded, wait for the side stream on the host instead
    if (fork && (cudaEventRecord(s->join_ev, ys) != cudaSuccess ||
                 cudaStreamWaitEvent(cs, s->join_ev, 0) != cudaSuccess))
      cudaStreamSynchronize(ys);
    trace_begin(s, k_u);
    float *qtf = nullptr, *primtf = nullptr;
    if constexpr (std::is_same<T, float>::value) {
      qtf = W.qt;
      primtf = W.primt;
    }
    kh_update<T><<<unsigned((nc + 255) / 256), 256, 0, cs>>>(G, stage, W.fx, W.fy, s->q, s->q0,
                                                            s->v, s->v0, W.vt, s->w, s->w0, W.wt,
                                                            W.prim, qtf, primtf, s->dstate);
    trace_end(s);
  }
  k_end_step<<<1, 1, 0, cs>>>(s->dstate);
}

}  // namespace
}  // namespace hteno
