// Conversions and the SSP-RK3 stage for the mixed-precision kernels (float reconstruction and
// fluxes, double state).  On GB300 the FP64 pipe, which also executes the hardware float <->
// double conversions, runs at 1/64 of the FP32 rate; these conversions run on the integer pipes.
#pragma once

namespace hteno {
namespace mix {

// Double -> float and float -> double on the integer pipes: the same results as the hardware
// conversions (round to nearest even) for normal numbers, infinities and NaN; subnormal results
// are flushed to signed zero.
__device__ __forceinline__ float d2f(double d) {
  const unsigned hi = unsigned(__double2hiint(d)), lo = unsigned(__double2loint(d));
  const unsigned s = hi & 0x80000000u;
  const unsigned eb = (hi >> 20) & 0x7ffu;
  const int e = int(eb) - 896;  // float biased exponent
  unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29);
  const unsigned rest = lo & 0x1fffffffu;
  m += (rest > 0x10000000u || (rest == 0x10000000u && (m & 1u))) ? 1u : 0u;
  if (eb == 0x7ffu) return __uint_as_float(s | 0x7f800000u | (((hi & 0xfffffu) | lo) ? 0x400000u : 0u));
  if (e <= 0) return __uint_as_float(s);
  if (e >= 255) return __uint_as_float(s | 0x7f800000u);
  return __uint_as_float(s | ((unsigned(e) << 23) + m));  // a mantissa carry bumps the exponent
}
__device__ __forceinline__ double f2d(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned s = u & 0x80000000u, e = (u >> 23) & 0xffu, m = u & 0x7fffffu;
  if (e == 0) return __hiloint2double(int(s), 0);
  const unsigned e2 = e == 255u ? 2047u : e + 896u;
  return __hiloint2double(int(s | (e2 << 20) | (m >> 3)), int(m << 29));
}

// SSP-RK3 stage (Schemes_SSPRK.cpp:3-15) in double with fused multiply-adds (the mixed path does
// not need the reference's rounding sequence, only FP64 accumulation).  The factors come from memory
// and the product is written as a fused multiply-add: the FP64 unit takes 64 cycles per warp for a
// fused multiply-add of three vector registers and 76 for one with a literal or for a multiplication.
struct RkStage {
  double dt, a, b, one, nzero;  // q = a (qn + dt rhs) + b q0; 1, -0
  int stage;
  __device__ __forceinline__ double operator()(double q0, double qn, double rhs) const {
    if (stage == 1) return fma(dt, rhs, q0);
    return fma(a, fma(dt, rhs, qn), fma(b, q0, nzero));
  }
};
static __device__ double g_rk[6] = {0.25, 0.75, 2.0 / 3.0, 1.0 / 3.0, 1.0, -0.0};
__device__ __forceinline__ double ld_factor(int k) {
  double r;
  asm("ld.global.nc.f64 %0, [%1];" : "=d"(r) : "l"(__cvta_generic_to_global(g_rk + k)));
  return r;
}
__device__ __forceinline__ RkStage rk_stage(int stage, double dt) {
  const int k = stage == 2 ? 0 : 2;
  return RkStage{dt, ld_factor(k), ld_factor(k + 1), ld_factor(4), ld_factor(5), stage};
}

// d = a - b, true where that is the exact difference: the two are within a factor of two (so |a - b| is
// at most the smaller of them) and it is not subnormal, which f2d flushes.
__device__ __forceinline__ bool exact_diff(float a, float b, float* d) {
  *d = a - b;
  const float m = fabsf(*d);
  return m <= fminf(fabsf(a), fabsf(b)) && (m >= 1.17549435e-38f || m == 0.0f);
}

// The largest wave speed max(u - c, |u + c|, v - c, |v + c|) of a new state, in double (timeStepping,
// FV_System2D.cpp:622-633): the first dt.  Only the maximum matters, so a cell is evaluated in double
// (divisions and square roots, ~3000 cycles of the FP64 pipe a warp) only where a float upper bound of
// its speed is not below the largest speed known (the block's own and, once an iteration, the grid's),
// and where it is not the cell that its thread evaluated last (regions at the largest speed): the same
// bits as evaluating all.  Each block takes a contiguous share of the cells, so that the first
// iteration samples the whole grid.  The bound holds for any input: a float operation is off by less
// than 2^-22 of its result or 2^-126, and the terms 1e-5, 1.0001, 1e-36 are far above the sum of
// these; NaN and infinities are evaluated.
// k_max_speed of 4096^2 cells: 1.46 -> 0.35 ms (reading memory: 0.08).
struct SpeedFilter {
  unsigned long long* maxbits;  // global: bits of the largest speed found by any block
  unsigned* found;              // shared: bits of a float below the largest speed known
  float g1, gamma;
  double last[4];  // conserved variables that this thread evaluated last
  size_t k, end;   // this thread's next cell (step blockDim.x) and the end of the block's share
  // every thread of the block calls it
  __device__ __forceinline__ SpeedFilter(unsigned* f, unsigned long long* bits, double g1d, double gammad, size_t nc)
      : maxbits(bits), found(f), g1(fabsf(float(g1d))), gamma(fabsf(float(gammad))), last{0.0, 0.0, 0.0, 0.0} {
    if (threadIdx.x == 0) *found = 0u;
    __syncthreads();
    const size_t share = (nc + gridDim.x - 1) / gridDim.x;
    const size_t lo = min(nc, blockIdx.x * share);
    end = min(nc, lo + share);
    k = lo + threadIdx.x;
  }
  static __device__ __forceinline__ unsigned below(double speed) {  // 0 for NaN, negative and huge ones
    const float low = d2f(speed) * 0.9999f;
    return low > 0.0f && low <= 3e38f ? __float_as_uint(low) : 0u;
  }
  __device__ __forceinline__ bool may_exceed(const double* q) const {
    if (threadIdx.x == 0)
      atomicMax(found, below(__longlong_as_double(*static_cast<volatile unsigned long long*>(maxbits))));
    const float r = d2f(q[0]), mx = d2f(q[1]), my = d2f(q[2]), e = d2f(q[3]);
    const float ir = __frcp_rn(fminf(fabsf(r), 1e30f));
    const float au = fabsf(mx) * ir, av = fabsf(my) * ir;
    const float ke = 0.5f * (fabsf(mx) * au + fabsf(my) * av);
    const float p = (fabsf(e - copysignf(ke, r)) + 1e-5f * (fabsf(e) + ke) + 1e-36f) * g1;
    const float bound = (fmaxf(au, av) + sqrtf(gamma * p * ir + 1e-36f) + 1e-36f * ir) * 1.0001f;
    if (bound < __uint_as_float(*static_cast<volatile unsigned*>(found))) return false;
    long long d = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) d |= __double_as_longlong(q[k]) ^ __double_as_longlong(last[k]);
    return d != 0;  // (the first `last` is 0 / 0: a speed that is NaN and counts for nothing)
  }
  __device__ __forceinline__ void add(const double* q, double speed) {
    const unsigned low = below(speed);
    if (atomicMax(found, low) < low) atomicMax(maxbits, static_cast<unsigned long long>(__double_as_longlong(speed)));
#pragma unroll
    for (int k = 0; k < 4; ++k) last[k] = q[k];
  }
};

}  // namespace mix
}  // namespace hteno
