// FP64 arithmetic in three-register form.
//
// GB300's FP64 units take one warp instruction per 64 cycles and SM sub-partition when it is a
// fused multiply-add of three vector registers, and one per 76 cycles when it is an addition, a
// multiplication, or a fused multiply-add with an immediate, constant-bank or uniform operand
// (measured with all four sub-partitions issuing: chains of a*b+c in registers 64.1, additions and
// multiplications 76.1, a*b+c with one literal 76.3 cycles per warp instruction).  The
// bit-reproducible kernels are bound by that unit and are mostly additions and multiplications,
// so they are written as fused multiply-adds that round to the same bits:
//
//   a + b = fma(a, 1, b)      the product is exact
//   a * b = fma(a, b, -0)     adding -0 changes neither a rounded product nor the sign of a zero
//   k x + y, k a power of two = fma(k, x, y)   the product is exact: one operation instead of two
//                              (k < 1 only where a subnormal k x does not reach a result)
//
// 1, -0 and every literal come from a table in global memory, so that they sit in vector
// registers (a literal the compiler sees would go back into the instruction or to a uniform
// register).  Overflow, infinities and NaN go as in the separate operations, except where a power-of-two
// product would overflow by itself (|x| above 2^1021: in the indicators, whose squares then overflow too).  Measured, the same bits:
// two FV 2D steps at 1024^2 with state copies 56.9 -> 50.6 ms, four periodic teno5i steps at
// 333 x 257 12.8 -> 11.4 ms, two Hermite 2D steps at 300 x 211 30.7 -> 23.2 ms, 96 steps of a 1D
// tube of 400 cells 9.35 -> 7.98 ms.
#pragma once

#include <cuda_runtime.h>

namespace hteno {
namespace par {

enum Lit : int {
  kOne, kNegZero, kHalf, kNegHalf, kQuarter, kNegQuarter, kThreeQuarters, kThreeHalves, kTwo, kNegTwo, kThree,
  kFour, kNegFour, kSix, kThirteenTwelfths, kEpsz, kEps6, k6908, k51001, k67923, k38947, k8209, k104963,
  k299076, k179098, k231153, kDiv5040, kDiv5040Lo, kDiv6, kDiv6Lo, kDiv24, kDiv24Lo, kDiv3, kDiv3Lo, k23, k26,
  // Schemes::Hermite's full-stencil indicators
  k1029270, k2129184, k1099914, k281121, k494958, k1099445, k4317056, k2118166, kDiv6720, kDiv6720Lo, k3156862, k13189240,
  k1710479, k9617754, k531552, k10149306, k26511200, k39700440, k15136011, k1076544, k29195478, kDiv1680, kDiv1680Lo,
  kLw0, kLw1, kRcpLw0, kLw1OverLw0,
  kLitCount
};
static __device__ double g_lit[kLitCount] = {
    1.0, -0.0, 0.5, -0.5, 0.25, -0.25, 0.75, 1.5, 2.0, -2.0, 3.0,
    4.0, -4.0, 6.0, 13.0 / 12.0, 1e-40, 1e-6, 6908.0, 51001.0, 67923.0, 38947.0, 8209.0, 104963.0,
    299076.0, 179098.0, 231153.0, 1.0 / 5040.0, 0x1.a01a01a01a01ap-73, 1.0 / 6.0, 0x1.5555555555555p-57,
    1.0 / 24.0, 0x1.5555555555555p-59, 1.0 / 3.0, 0x1.5555555555555p-56, 23.0, 26.0,
    1029270.0, 2129184.0, 1099914.0, 281121.0, 494958.0, 1099445.0, 4317056.0, 2118166.0, 1.0 / 6720.0,
    -0x1.fb1fb1fb1fb20p-67, 3156862.0,
    13189240.0, 1710479.0, 9617754.0, 531552.0, 10149306.0, 26511200.0, 39700440.0, 15136011.0, 1076544.0,
    29195478.0, 1.0 / 1680.0, -0x1.fb1fb1fb1fb20p-65, 1.0 - 2e-5, 1e-5, 1.0 / (1.0 - 2e-5), 1e-5 / (1.0 - 2e-5)};

// A double of global memory that is constant while the kernel runs, in a vector register.
__device__ __forceinline__ double ldk(const double& x) {
  double r;
  asm("ld.global.nc.f64 %0, [%1];" : "=d"(r) : "l"(__cvta_generic_to_global(&x)));
  return r;
}

// A double whose + - * are the forms above.
struct fp {
  double v;
  __device__ __forceinline__ fp() {}
  __device__ __forceinline__ fp(double x) : v(x) {}
};
__device__ __forceinline__ fp lit(Lit k) { return fp(ldk(g_lit[k])); }
__device__ __forceinline__ fp operator+(fp a, fp b) { return fma(a.v, lit(kOne).v, b.v); }
__device__ __forceinline__ fp operator-(fp a, fp b) { return fma(-b.v, lit(kOne).v, a.v); }
__device__ __forceinline__ fp operator*(fp a, fp b) { return fma(a.v, b.v, lit(kNegZero).v); }
__device__ __forceinline__ fp operator-(fp a) { return fp(-a.v); }
// k x + y for a power of two k (also 0): the product is exact
__device__ __forceinline__ fp scaled(Lit k, fp x, fp y) { return fma(x.v, lit(k).v, y.v); }
__device__ __forceinline__ fp abs_(fp a) { return fp(fabs(a.v)); }

}  // namespace par
}  // namespace hteno
