// Two floats per instruction: sm_100's packed add, mul and fma on a 64-bit register pair, each half
// rounded to nearest as the scalar instruction rounds it (subnormals kept).  The packed fma takes the
// FMA pipe as long as two scalar ones but one issue slot instead of two: on GB300 chains of four ran
// at 2.0 cycles per packed and 1.1 per scalar warp instruction and sub-partition.  In the fused mixed
// FV 2D stage (issue-bound: 60 % of the slots with the FMA pipe 41 % busy) the two sides of a
// reconstruction, of GL3 and of the flux, and neighbouring cells of the projection, in pairs: 303 -> 241
// us per stage of 1024^2 (32 x 16 tiles, three blocks per SM), the same bits.
#pragma once

#include <cuda_runtime.h>

namespace hteno {

struct f2 {
  unsigned long long b;
};
__device__ __forceinline__ f2 pack(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f2 dup(float x) { return pack(x, x); }
__device__ __forceinline__ float lo(f2 a) {
  float l, h;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(l), "=f"(h) : "l"(a.b));
  return l;
}
__device__ __forceinline__ float hi(f2 a) {
  float l, h;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(l), "=f"(h) : "l"(a.b));
  return h;
}
__device__ __forceinline__ f2 mad(f2 a, f2 b, f2 c) {  // a * b + c, rounded once
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(a.b), "l"(b.b), "l"(c.b));
  return r;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ f2 operator+(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ f2 operator-(f2 a, f2 b) { return mad(b, dup(-1.0f), a); }  // the product is exact
__device__ __forceinline__ f2 operator-(f2 a) {
  return f2{a.b ^ 0x8000000080000000ull};
}
__device__ __forceinline__ f2 abs_(f2 a) { return f2{a.b & 0x7fffffff7fffffffull}; }
// x0 y0 + x1 y1 + x2 y2, summed left to right
__device__ __forceinline__ f2 dot3m(f2 x0, f2 y0, f2 x1, f2 y1, f2 x2, f2 y2) { return mad(x2, y2, mad(x1, y1, x0 * y0)); }

}  // namespace hteno
