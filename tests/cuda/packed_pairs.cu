// The packed float functions of the mixed FV 2D and Hermite 2D kernels beside the scalar functions that the
// pointwise entry points run (and test): the number of outputs whose bits differ, over stencils and states of
// many shapes, the two halves of every pair different.  Compiled twice, as the solvers' units are: FV
// (UNIT 0) without implicit contraction, Hermite (UNIT 1) with it.  See tests/test_gpu_packed_pairs.py.
#include "../../hermite-teno_gb300/csrc/fv2d_fused.cuh"
#include "../../hermite-teno_gb300/csrc/hermite_math.cuh"

using namespace hteno;

namespace {

__constant__ DevConst c_dev;
constexpr int kIn = 15, kOut = 12, kThreads = 128;

__device__ unsigned long long next(unsigned long long& s) {
  s += 0x9e3779b97f4a7c15ull;
  unsigned long long z = s;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
__device__ float uni(unsigned long long& s) { return float(next(s) >> 40) * 5.9604645e-8f; }

// 6 cell values u and 4 derivatives d of the shape `kind`
__device__ void stencil(unsigned long long& s, int kind, float rdif, float* u, float* d) {
  const float base = 2.f * uni(s) - 1.f, g = (uni(s) - 0.5f) * exp2f(-8.f * uni(s)), z = exp2f(-12.f * uni(s));
  const float ph = 6.28f * uni(s), jump = 4.f * uni(s) - 2.f;
  const int at = int(next(s) % 6);
  float scale = 1.f;
  if (kind == 5) scale = exp2f(-100.f - 49.f * uni(s));  // tiny, down to subnormals
  if (kind == 6) scale = exp2f(20.f + 45.f * uni(s));    // huge: squares overflow
  for (int k = 0; k < 6; ++k) {
    u[k] = kind == 4 ? base : base + g * k + z * __sinf(ph + k) + (kind == 1 ? 0.01f * (uni(s) - 0.5f) : 0.f);
    if (kind == 3 && k >= at) u[k] += jump;
    u[k] *= scale;
  }
  for (int k = 0; k < 4; ++k) {
    d[k] = kind == 4 ? 0.f : (g + z * __cosf(ph + k) + (kind == 1 ? 0.01f * (uni(s) - 0.5f) : 0.f)) * rdif;
    d[k] *= scale;
  }
  if (kind == 7) u[at] = next(s) & 1 ? __int_as_float(0x7fc00000) : __int_as_float(0x7f800000);
}
__device__ void state(unsigned long long& s, int kind, float* q) {
  const float rho = kind == 5 ? exp2f(-30.f * uni(s)) : 0.1f + 3.f * uni(s);
  const float m = kind == 2 ? 6.f : 1.f, u = m * (2.f * uni(s) - 1.f), v = m * (2.f * uni(s) - 1.f);
  const float p = kind == 6 ? -uni(s) : 0.05f + uni(s);
  q[0] = rho;
  q[1] = rho * u;
  q[2] = rho * v;
  q[3] = p / 0.4f + 0.5f * rho * (u * u + v * v);
  if (kind == 7) q[next(s) % 4] = __int_as_float(0x7fc00000);
}
__device__ Roe2<float> roe_of(const float* a, const float* b) {
  float w[2][4], h[2];
  for (int k = 0; k < 2; ++k) {
    const float* q = k ? b : a;
    w[k][1] = q[1] / q[0];
    w[k][2] = q[2] / q[0];
    w[k][3] = (q[3] - 0.5f * (q[1] * w[k][1] + q[2] * w[k][2])) * 0.4f;
    h[k] = (q[3] + w[k][3]) / q[0];
  }
  return roe2<float>(0.4f, sqrtf(fabsf(a[0])), w[0][1], w[0][2], h[0], sqrtf(fabsf(b[0])), w[1][1], w[1][2], h[1]);
}

// faces 0: in = u[6], d[4]; else a Roe average [7] and two states' values [8]: characteristic ones of direction
// 1 or 2 (faces 1, 2) or conserved ones (3)
__global__ void generate(int faces, float rdif, unsigned long long seed, float* in, long n) {
  const long i = blockIdx.x * long(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  unsigned long long s = seed * 0x2545f4914f6cdd1dull + i;
  const int kind = int(next(s) % 8);
  float x[kIn] = {};
  if (faces == 0) {
    stencil(s, kind, rdif, x, x + 6);
  } else {
    float ql[4], qr[4];
    state(s, kind, ql);
    state(s, kind == 4 ? 0 : kind, qr);
    if (kind == 4)
      for (int k = 0; k < 4; ++k) qr[k] = ql[k];
    const Roe2<float> R = roe_of(ql, qr);
    const float r[7] = {R.vxm, R.vym, R.hm, R.qm, R.cm, R.rcm, R.b1};
    for (int k = 0; k < 7; ++k) x[k] = r[k];
    if (faces <= 2) {  // which R takes back to about the states
      roe_left(R, faces, ql, x + 7);
      roe_left(R, faces, qr, x + 11);
    } else {
      for (int k = 0; k < 4; ++k) x[7 + k] = ql[k], x[11 + k] = qr[k];
    }
  }
  for (int k = 0; k < kIn; ++k) in[k * n + i] = x[k];
}

struct Args {
  HermiteK<float> K;
  const float* in;
  float* out;
  long n;
  __device__ void load(long i, float* x) const {
    for (int k = 0; k < kIn; ++k) x[k] = in[k * n + i];
  }
  __device__ void store(long i, int k, float x) const { out[k * n + i] = x; }
};
__device__ Roe2<float> roe_in(const float* x) { return Roe2<float>{x[0], x[1], x[2], x[3], x[4], x[5], x[6]}; }

// What is compared.  scalar() takes one sample, packed() the samples i and i + 1.
enum What { kTeno5, kTeno5i, kRouted, kRoutedMinus, kOther2, kOther3, kOther4, kOther5, kOther6, kOther7, kGl3, kLeft1,
            kLeft2, kRight1, kRight2, kHllc1, kHllc2, kRusanov1, kRusanov2, kHteno, kTenoCross, kCount };

__global__ void __launch_bounds__(kThreads) scalar(int what, Args a) {
  const long i = blockIdx.x * long(blockDim.x) + threadIdx.x;
  if (i >= a.n) return;
  float x[kIn], o[8] = {};
  a.load(i, x);
  int nout = 2;
  if (what <= kTeno5i || what == kTenoCross) {
    lagrange_recon(c_dev, what == kTeno5i ? 1 : 0, x, o[0], o[1]);
  } else if (what == kRouted || what == kRoutedMinus) {
    float t[2];
    lagrange_recon(c_dev, 2, x, o[0], o[1]);
    lagrange_recon(c_dev, 0, x, t[0], t[1]);
    o[0] = catchnan(o[0]);
    o[1] = what == kRouted ? catchnan(o[1]) : t[1];
  } else if (what <= kOther7) {
    lagrange_recon(c_dev, what - kOther2 + 2, x, o[0], o[1]);
  } else if (what == kGl3) {
    gl3(c_dev, x, o[0], o[1], o[2]);
    nout = 3;
  } else if (what == kHteno) {
    hermite_recon(c_dev, a.K, 0, x, x + 6, o);
    nout = 4;
  } else {
    const Roe2<float> R = roe_in(x);
    const int dir = (what - kLeft1) % 2 + 1;
    nout = what <= kRight2 ? 8 : 4;
    if (what <= kLeft2) {
      roe_left(R, dir, x + 7, o);
      roe_left(R, dir, x + 11, o + 4);
    } else if (what <= kRight2) {
      roe_right(R, dir, x + 7, o);
      roe_right(R, dir, x + 11, o + 4);
    } else {
      float ql[4], qr[4];
      roe_right(R, dir, x + 7, ql);
      roe_right(R, dir, x + 11, qr);
      if (what <= kHllc2) hllc2(0.4f, dir, ql, qr, o);
      else rusanov2(1.4f, 0.4f, dir, R, ql, qr, o);
    }
  }
  for (int k = 0; k < nout; ++k) a.store(i, k, o[k]);
}

__global__ void __launch_bounds__(kThreads) packed(int what, Args a) {
#if UNIT == 0
  __shared__ float tab[2][8][3];
  if (threadIdx.x < 48) {
    const int side = threadIdx.x / 24, pat = threadIdx.x % 24 / 3, k = threadIdx.x % 3;
    tab[side][pat][k] = side ? c_dev.f_wtab_p[pat][k] : c_dev.f_wtab_m[pat][k];
  }
  __syncthreads();
#else
  __shared__ HermiteTab tab;
  load_hermite_tab(tab, a.K, c_dev);
#endif
  const long i = blockIdx.x * long(blockDim.x) + threadIdx.x;
  if (i >= a.n) return;
  float x[kIn], y[kIn];
  a.load(i, x);
  a.load(i ^ 1, y);  // (n is even)
  if (what == kGl3) {
    const Gl3f g = gl3_pair<UNIT == 1>(c_dev, pack(x[0], y[0]), pack(x[1], y[1]), pack(x[2], y[2]), pack(x[3], y[3]),
                                       pack(x[4], y[4]));
    const f2 o[3] = {g.a, g.b, g.c};
    for (int k = 0; k < 3; ++k) {  // the low half here, the high half's partner in the rows behind
      a.store(i, k, lo(o[k]));
      a.store(i ^ 1, 3 + k, hi(o[k]));
    }
    return;
  }
  const f2 P0 = pack(x[0], x[1]), P1 = pack(x[2], x[3]), P2 = pack(x[4], x[5]);
  if (what >= kLeft1 && what <= kRusanov2) {
    const Roe2<float> R = roe_in(x);
    const int dir = (what - kLeft1) % 2 + 1;
    f2 c[4], o[4];
    for (int k = 0; k < 4; ++k) c[k] = pack(x[7 + k], x[11 + k]);
    if (what <= kRight2) {
      if (what <= kLeft2) project2(left_rows(R, dir), dir, c, o);
      else right2(R, dir, c, o);
      for (int k = 0; k < 4; ++k) {
        a.store(i, k, lo(o[k]));
        a.store(i, 4 + k, hi(o[k]));
      }
    }
#if UNIT == 0
    if (what > kRight2) {
      const int flux = what <= kHllc2 ? HTENO_FLUX_HLLC : HTENO_FLUX_RUSANOV;
      const fused::F4 F = dir == 1 ? fused::gauss_flux<1>(R, flux, 0.4f, 1.4f, c[0], c[1], c[2], c[3])
                                   : fused::gauss_flux<2>(R, flux, 0.4f, 1.4f, c[0], c[1], c[2], c[3]);
      for (int k = 0; k < 4; ++k) a.store(i, k, F.v[k]);
    }
#endif
    return;
  }
#if UNIT == 0
  fused::Sides o;
  if (what <= kTeno5i) o = fused::teno_sides(c_dev, what == kTeno5i, tab, P0, P1, P2, 0, false);
  else if (what <= kRoutedMinus) o = fused::teno_sides(c_dev, false, tab, P0, P1, P2, what == kRouted ? 3 : 1, false);
  else o = fused::other_sides(c_dev, what - kOther2 + 2, tab, x[0], x[1], x[2], x[3], x[4], x[5]);
  a.store(i, 0, o.m);
  a.store(i, 1, o.p);
#else
  if (what == kHteno) {
    const HtenoSides h = hteno_sides(tab, a.K.dif, P0, P1, pack(x[6], x[7]), pack(x[8], x[9]));
    const f2 o[2] = {h.u, h.d};
    for (int k = 0; k < 2; ++k) {
      a.store(i, 2 * k, lo(o[k]));
      a.store(i, 2 * k + 1, hi(o[k]));
    }
  } else {
    const f2 u = teno5_sides(c_dev, tab, P0, P1, P2);
    a.store(i, 0, lo(u));
    a.store(i, 1, hi(u));
  }
#endif
}

// outputs k of `a` against outputs k and (twice) k + nout of `b`
__global__ void compare(const float* a, const float* b, int nout, int twice, long n, unsigned long long* bad) {
  const long i = blockIdx.x * long(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  unsigned m = 0;
  for (int k = 0; k < nout; ++k)
    for (int t = 0; t <= twice; ++t) {
      const float x = a[k * n + i], y = b[(k + t * nout) * n + i];
      m += !(__float_as_uint(x) == __float_as_uint(y) || (isnan(x) && isnan(y)));
    }
  if (m) atomicAdd(bad, (unsigned long long)m);
}

}  // namespace

// Outputs of `what` over n (even) samples whose bits differ, or a negative CUDA error.
extern "C" long packed_mismatches(int what, long n, unsigned long long seed) {
  DevConst h;
  fill_dev_const(&h);
  float *in = nullptr, *o1 = nullptr, *o2 = nullptr;
  unsigned long long *bad = nullptr, result = 0;
  const unsigned blocks = unsigned((n + kThreads - 1) / kThreads);
  const HermiteK<float> K = make_hermite_k<float>(1.0 / 2048 * 1.1);
  const int faces = what >= kLeft1 && what <= kRusanov2 ? (what <= kLeft2 ? 3 : (what - kLeft1) % 2 + 1) : 0;
  const int nout = what == kGl3 ? 3 : what == kHteno ? 4 : !faces ? 2 : what <= kRight2 ? 8 : 4;
  cudaError_t e = cudaMemcpyToSymbol(c_dev, &h, sizeof(h));
  if (e == cudaSuccess) e = cudaMalloc(&in, kIn * n * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&o1, kOut * n * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&o2, kOut * n * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&bad, sizeof(*bad));
  if (e == cudaSuccess) e = cudaMemset(bad, 0, sizeof(*bad));
  if (e == cudaSuccess) {
    generate<<<blocks, kThreads>>>(faces, float(K.rdif), seed, in, n);
    scalar<<<blocks, kThreads>>>(what, Args{K, in, o1, n});
    packed<<<blocks, kThreads>>>(what, Args{K, in, o2, n});
    compare<<<blocks, kThreads>>>(o1, o2, nout, what == kGl3, n, bad);
    e = cudaMemcpy(&result, bad, sizeof(result), cudaMemcpyDeviceToHost);
  }
  cudaFree(in);
  cudaFree(o1);
  cudaFree(o2);
  cudaFree(bad);
  return e == cudaSuccess ? long(result) : -long(e);
}
