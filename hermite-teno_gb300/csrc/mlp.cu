// Learned stencil classifier: a 6 -> 32 -> 32 -> 3 MLP (ReLU, sigmoid outputs) that predicts the
// three TENO5 cut-off bits of a normalised 6-cell characteristic stencil (cutOff,
// Schemes_Lagrange.cpp:1141-1149, on the left-biased side; the right side is the mirrored
// stencil).  BF16 operands, FP32 accumulation, on the tcgen05 tensor cores:
//
//   forward   D1 = X W1^T, H1 = relu(D1 + b1); D2 = H1 W2^T, H2 = relu(D2 + b2);
//             D3 = H2 W3^T, p = sigmoid(D3 + b3)
//   backward  dZ3 = (p - y) / n;  dH2 = dZ3 W3;  dZ2 = dH2 * [H2 > 0];  dH1 = dZ2 W2;
//             dZ1 = dH1 * [H1 > 0];  dW3 += dZ3^T H2, dW2 += dZ2^T H1, dW1 += dZ1^T X
//
// One CTA of 128 threads owns a 128-row tile (thread = row = tensor-memory lane); weight
// gradients accumulate in tensor memory across the CTA's tiles and are added to the global
// gradient at the end.  Adam runs on FP32 master weights; the kernels read BF16 images of them.
// No reference counterpart: the reference has no learned component (its precedent is the LMPE
// troubled-cell sensor of FVHermite_System1D.cpp:239-290).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <random>
#include <vector>

#include "fv2d_fused.cuh"
#include "hteno_internal.h"
#include "launch.cuh"
#include "mlp_internal.cuh"

struct hteno_mlp;

namespace hteno {
namespace mlp {
namespace {

constexpr uint32_t kWaitLimit = 1u << 22;  // polls of an mbarrier before giving up

// Training, one tile of 128 rows at a time.  The transposed operands (rows = features or outputs,
// K = the tile's rows) have their core matrices kTK = 144 bytes apart along K instead of 128: eight
// consecutive rows write one 16-byte line of each core matrix, and with 128 the four core matrices
// that a warp writes would fall on the same banks.
constexpr int kTK = 144, kTGroup = 16 * kTK;  // bytes per core matrix along K, per group of 8 rows
struct Smem {
  // A operand of the weight gradients: 32 outputs.  The products read 128 rows (9 KB further each
  // 32): what lies there goes to accumulator rows that nothing reads.
  alignas(128) unsigned char at[4 * kTGroup];
  alignas(128) unsigned char x[128 * 16 * 2];
  alignas(128) unsigned char xt[2 * kTGroup];
  alignas(128) unsigned char h1[128 * 32 * 2];
  alignas(128) unsigned char h1t[4 * kTGroup];
  alignas(128) unsigned char h2[128 * 32 * 2];
  alignas(128) unsigned char h2t[4 * kTGroup];
  alignas(128) unsigned char dz3[128 * 16 * 2];
  alignas(128) unsigned char dz2[128 * 32 * 2];
  alignas(128) unsigned char w1[32 * 16 * 2];
  alignas(128) unsigned char w2[32 * 32 * 2];
  alignas(128) unsigned char w3[16 * 32 * 2];
  alignas(128) unsigned char w3t[32 * 16 * 2];
  alignas(128) unsigned char w2t[32 * 32 * 2];
  float b1[32], b2[32], b3[16];
  // bias gradients and loss, one slot per warp (summed in warp order at the end: deterministic)
  float gb1[4][32], gb2[4][32], gb3[4][4];
  float loss[4];
  alignas(8) uint64_t mbar;
  uint32_t tmem;
  static constexpr bool kTrain = true;
  static constexpr uint32_t kTmemCols = 256;
};
static_assert(sizeof(Smem) >= 16 * kTGroup, "the A operand's 128 rows lie inside the structure");

// Shared memory of the inference kernels (the forward pass only).  A CTA runs kCT tiles of 128
// rows at once, so that each issue-wait-load round trip of a layer serves 512 rows; a tile's X,
// H1 and H2 share one buffer (each is dead once the product that reads it has completed), and its
// three accumulators share 32 tensor-memory columns.  The allocation is padded to 48 KB so that at
// most 4 CTAs share an SM, whose 4 x 128 tensor-memory columns are the SM's 512.
constexpr int kCT = 4;              // tiles per network round
constexpr int kCRound = kCT * 128;  // rows per network round
struct SmemC {
  alignas(128) unsigned char buf[kCT][128 * 32 * 2];
  alignas(128) unsigned char w1[32 * 16 * 2];
  alignas(128) unsigned char w2[32 * 32 * 2];
  alignas(128) unsigned char w3[16 * 32 * 2];
  alignas(8) float b1[32], b2[32], b3[16];
  alignas(8) uint64_t mbar;
  uint32_t tmem;
  static constexpr bool kTrain = false;
  static constexpr uint32_t kTmemCols = 128;
};
constexpr size_t kSmemCBytes = 48 * 1024;
static_assert(sizeof(SmemC) <= kSmemCBytes, "inference shared memory");

// tensor-memory columns
constexpr uint32_t C_D1 = 0, C_D2 = 32, C_D3 = 64, C_DH2 = 80, C_DH1 = 112;
constexpr uint32_t C_GW3 = 144, C_GW2 = 176, C_GW1 = 208;

__device__ __forceinline__ uint64_t desc_k(const unsigned char* base, int K, int kstep) {
  return tc::sdesc(tc::smem_u32(base) + uint32_t(kstep) * 256u, 128u, uint32_t(K / 8) * 128u);
}

// Transposed operand: byte offset of (r, k), and the descriptor of K step kstep (16 of K).
__device__ __forceinline__ uint32_t tmaj(int r, int k) {
  return uint32_t((r >> 3) * kTGroup + (k >> 3) * kTK + (r & 7) * 16 + (k & 7) * 2);
}
__device__ __forceinline__ uint64_t desc_t(const unsigned char* base, int kstep) {
  return tc::sdesc(tc::smem_u32(base) + uint32_t(kstep) * 2u * kTK, kTK, kTGroup);
}

// Row-major BF16 [rows][K] image to the operand layout, 16 bytes (8 of K) at a time.
__device__ __forceinline__ void put_image(unsigned char* dst, const void* img, int rows, int K) {
  for (int e = threadIdx.x; e < rows * K / 8; e += blockDim.x) {
    const int r = e / (K / 8), g = e % (K / 8);
    *reinterpret_cast<uint4*>(dst + tc::kmaj(r, 8 * g, K)) = static_cast<const uint4*>(img)[e];
  }
}

// Copies the BF16 weight images into the operand layouts and the FP32 biases.
template <typename SM>
__device__ void load_weights(SM& S, const Weights& W) {
  put_image(S.w1, W.w1, 32, 16);
  put_image(S.w2, W.w2, 32, 32);
  put_image(S.w3, W.w3, 16, 32);
  if constexpr (SM::kTrain) {
    put_image(S.w3t, W.w3t, 32, 16);
    put_image(S.w2t, W.w2t, 32, 32);
  }
  for (int e = threadIdx.x; e < 32; e += blockDim.x) {
    S.b1[e] = W.b1[e];
    S.b2[e] = W.b2[e];
    if (e < 16) S.b3[e] = W.b3[e];
  }
}

// Issue (thread 0) after a barrier; every thread then waits for completion.  Returns false on
// timeout (uniform over the block).
template <typename SM>
__device__ __forceinline__ bool wait_mma(SM& S, uint32_t& phase, uint32_t limit) {
  const bool ok = !__syncthreads_or(!tc::mbar_wait(&S.mbar, phase, limit));
  if (ok) phase ^= 1u;  // on timeout `phase` stays the pending one
  tc::fence_after();
  return ok;
}

__device__ __forceinline__ void before_issue() {
  tc::fence_proxy_async();
  tc::fence_before();
  __syncthreads();
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The sums over the warp of each of 32 columns, lane c's result being column c's: halves of the
// columns change sides at each step, 31 shuffles instead of 160 for 32 warp_sum, the same additions.
__device__ __forceinline__ float column_sums(float* v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < o; ++j) {
      const float send = up ? v[j] : v[j + o], keep = up ? v[j + o] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// Two floats -> two BF16 (round to nearest even), lo to the lower address; and back.
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// This thread's 32 values, packed in w, as row `row` of a K-major operand (dst, unless null) and as
// column `row` of a transposed one.
__device__ __forceinline__ void put_row32(unsigned char* dst, unsigned char* dst_t, int row, const uint32_t* w) {
  if (dst != nullptr) {
#pragma unroll
    for (int g = 0; g < 4; ++g)
      *reinterpret_cast<uint4*>(dst + tc::kmaj(row, 8 * g, 32)) =
          make_uint4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]);
  }
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    *reinterpret_cast<uint16_t*>(dst_t + tmaj(2 * c, row)) = uint16_t(w[c]);
    *reinterpret_cast<uint16_t*>(dst_t + tmaj(2 * c + 1, row)) = uint16_t(w[c] >> 16);
  }
}

// A hidden layer of this thread's row (training): bias and ReLU on the accumulator row at taddr, the
// BF16 operands of the next layer and of the weight gradient; returns where the ReLU passes.
__device__ __forceinline__ uint32_t hidden_train(uint32_t taddr, const float* b, unsigned char* dst,
                                                 unsigned char* dst_t, int row) {
  float h[32];
  tc::tmem_ld16(taddr, h);
  tc::tmem_ld16(taddr + 16, h + 16);
  uint32_t w[16], pass = 0u;
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    h[c] = fmaxf(h[c] + b[c], 0.0f);
    pass |= h[c] > 0.f ? 1u << c : 0u;
  }
#pragma unroll
  for (int c = 0; c < 16; ++c) w[c] = pack_bf16(h[2 * c], h[2 * c + 1]);
  put_row32(dst, dst_t, row, w);
  return pass;
}

// The error terms of a hidden layer: the accumulator row at taddr where the ReLU passed, as operands
// (dst may be null); returns this warp's sum of column `lane` of the rounded terms (bias gradient).
__device__ __forceinline__ float error_train(uint32_t taddr, uint32_t pass, unsigned char* dst,
                                             unsigned char* dst_t, int row) {
  float d[32];
  tc::tmem_ld16(taddr, d);
  tc::tmem_ld16(taddr + 16, d + 16);
  uint32_t w[16];
#pragma unroll
  for (int c = 0; c < 32; ++c) d[c] = (pass >> c) & 1u ? d[c] : 0.f;
#pragma unroll
  for (int c = 0; c < 16; ++c) w[c] = pack_bf16(d[2 * c], d[2 * c + 1]);
  put_row32(dst, dst_t, row, w);
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    d[2 * c] = bf_lo(w[c]);
    d[2 * c + 1] = bf_hi(w[c]);
  }
  return column_sums(d);
}

// Forward pass of the tile whose inputs are in S.x / S.xt: the logits z3 of this thread's row and
// where its two hidden layers' ReLUs pass; H1, H2 and their transposes stay in shared memory.
__device__ __forceinline__ bool forward(Smem& S, uint32_t tbase, uint32_t& phase, uint32_t* pass1,
                                        uint32_t* pass2, float* z3, uint32_t limit) {
  const int row = threadIdx.x;
  const uint32_t lane_addr = tbase + (uint32_t(threadIdx.x & ~31) << 16);
  before_issue();
  if (threadIdx.x == 0) {
    tc::fence_after();
    tc::mma_bf16(tbase + C_D1, desc_k(S.x, 16, 0), desc_k(S.w1, 16, 0), tc::idesc_bf16(128, 32), 0);
    tc::commit(&S.mbar);
  }
  if (!wait_mma(S, phase, limit)) return false;
  *pass1 = hidden_train(lane_addr + C_D1, S.b1, S.h1, S.h1t, row);
  before_issue();
  if (threadIdx.x == 0) {
    tc::fence_after();
    for (int s = 0; s < 2; ++s)
      tc::mma_bf16(tbase + C_D2, desc_k(S.h1, 32, s), desc_k(S.w2, 32, s), tc::idesc_bf16(128, 32), s);
    tc::commit(&S.mbar);
  }
  if (!wait_mma(S, phase, limit)) return false;
  *pass2 = hidden_train(lane_addr + C_D2, S.b2, S.h2, S.h2t, row);
  before_issue();
  if (threadIdx.x == 0) {
    tc::fence_after();
    for (int s = 0; s < 2; ++s)
      tc::mma_bf16(tbase + C_D3, desc_k(S.h2, 32, s), desc_k(S.w3, 32, s), tc::idesc_bf16(128, 16), s);
    tc::commit(&S.mbar);
  }
  if (!wait_mma(S, phase, limit)) return false;
  float d3[16];
  tc::tmem_ld16(lane_addr + C_D3, d3);
#pragma unroll
  for (int k = 0; k < 3; ++k) z3[k] = d3[k] + S.b3[k];
  return true;
}

// Two floats -> two BF16 (round to nearest even) with negative results clamped to +0: ReLU then
// rounding, in one instruction.  lo goes to the lower address.
__device__ __forceinline__ uint32_t pack_relu(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// Bias, ReLU and BF16 rounding of this thread's 32-column accumulator row, stored as its row of
// the next layer's A operand (four 16-byte rows of K-major core matrices).
__device__ __forceinline__ void hidden_row(uint32_t taddr, const float* b, unsigned char* dst, int row) {
  float h[32];
  tc::tmem_ld16(taddr, h);
  tc::tmem_ld16(taddr + 16, h + 16);
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = 8 * g + 2 * j;
      const f2 x = pack(h[c], h[c + 1]) + *reinterpret_cast<const f2*>(b + c);
      w[j] = pack_relu(lo(x), hi(x));
    }
    *reinterpret_cast<uint4*>(dst + tc::kmaj(row, 8 * g, 32)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// Forward pass of up to kCT tiles at once (inference): thread r holds row r of tile t in in[t]
// (6 BF16 features in .x .y .z); n valid rows in all, tiles beyond them are not computed.  Leaves
// the three output logits of each of its rows in z.  Returns false on a timed-out wait (uniform).
__device__ __forceinline__ bool forward_rows(SmemC& S, uint32_t tbase, uint32_t& phase, const uint4* in,
                                             int n, float (*z)[3], uint32_t limit) {
  const int row = threadIdx.x;
  const int ntile = (n + 127) >> 7;
  const uint32_t lane_addr = tbase + (uint32_t(threadIdx.x & ~31) << 16);
#pragma unroll
  for (int t = 0; t < kCT; ++t)
    if (t < ntile) {
      *reinterpret_cast<uint4*>(S.buf[t] + tc::kmaj(row, 0, 16)) = make_uint4(in[t].x, in[t].y, in[t].z, 0u);
      *reinterpret_cast<uint4*>(S.buf[t] + tc::kmaj(row, 8, 16)) = make_uint4(0u, 0u, 0u, 0u);
    }
  before_issue();
  if (threadIdx.x == 0) {
    tc::fence_after();
    for (int t = 0; t < ntile; ++t)
      tc::mma_bf16(tbase + 32 * t, desc_k(S.buf[t], 16, 0), desc_k(S.w1, 16, 0), tc::idesc_bf16(128, 32), 0);
    tc::commit(&S.mbar);
  }
  if (!wait_mma(S, phase, limit)) return false;
#pragma unroll
  for (int t = 0; t < kCT; ++t)
    if (t < ntile) hidden_row(lane_addr + 32 * t, S.b1, S.buf[t], row);
  before_issue();
  if (threadIdx.x == 0) {
    tc::fence_after();
    for (int t = 0; t < ntile; ++t)
      for (int k = 0; k < 2; ++k)
        tc::mma_bf16(tbase + 32 * t, desc_k(S.buf[t], 32, k), desc_k(S.w2, 32, k), tc::idesc_bf16(128, 32), k);
    tc::commit(&S.mbar);
  }
  if (!wait_mma(S, phase, limit)) return false;
#pragma unroll
  for (int t = 0; t < kCT; ++t)
    if (t < ntile) hidden_row(lane_addr + 32 * t, S.b2, S.buf[t], row);
  before_issue();
  if (threadIdx.x == 0) {
    tc::fence_after();
    for (int t = 0; t < ntile; ++t)
      for (int k = 0; k < 2; ++k)
        tc::mma_bf16(tbase + 32 * t, desc_k(S.buf[t], 32, k), desc_k(S.w3, 32, k), tc::idesc_bf16(128, 16), k);
    tc::commit(&S.mbar);
  }
  if (!wait_mma(S, phase, limit)) return false;
#pragma unroll
  for (int t = 0; t < kCT; ++t)
    if (t < ntile) {
      float d3[16];
      tc::tmem_ld16(lane_addr + 32 * t, d3);
#pragma unroll
      for (int k = 0; k < 3; ++k) z[t][k] = d3[k] + S.b3[k];
    }
  return true;
}

// Everything of a launch that does not need the weights.
template <typename SM>
__device__ void setup(SM& S) {
  if constexpr (SM::kTrain) {
    // the constant zeros of the operands: features 6..15 of X and X^T, outputs 3..15 of dZ3
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(S.x + tc::kmaj(threadIdx.x, 8, 16)) = zero;
    *reinterpret_cast<uint4*>(S.dz3 + tc::kmaj(threadIdx.x, 8, 16)) = zero;
    for (int e = threadIdx.x; e < 10 * 16; e += blockDim.x)
      *reinterpret_cast<uint4*>(S.xt + tmaj(6 + e / 16, 8 * (e % 16))) = zero;
    if (threadIdx.x < 16) S.gb3[threadIdx.x / 4][threadIdx.x % 4] = 0.f;
    if (threadIdx.x < 4) S.loss[threadIdx.x] = 0.f;
  }
  if (threadIdx.x == 0) {
    tc::mbar_init(&S.mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) tc::tmem_alloc(&S.tmem, SM::kTmemCols);
}
template <typename SM>
__device__ void setup(SM& S, const Weights& W) {
  setup(S);
  load_weights(S, W);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
}

template <typename SM>
__device__ void teardown(SM& S, uint32_t tbase) {
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (threadIdx.x < 32) tc::tmem_dealloc(tbase, SM::kTmemCols);
}

// Gradient of the mean BCE loss over `n_total` rows: each CTA writes its partial gradient (padded
// layout) to Gp[blockIdx.x] and its partial loss sum to Lp[blockIdx.x]; the next kernel adds the
// partials in CTA order, so the gradient does not depend on the order in which CTAs finish.  A batch
// is a tile or two per CTA, so the time is one tile's chain: six tensor-core round trips and the
// conversions between them, in one warp per scheduler.  Hence operand rows in 16-byte stores, the
// transposed ones without bank conflicts, bias gradients by column_sums, set-up and input loads
// before the previous kernel has completed.  Batches of 16384 rows, alone from cold caches: 16.3 -> 11.4
// us; a whole batch with its sums and update 34 -> 17.4 us.
// `limit`: polls of each tensor-core completion wait before the kernel gives up.
__global__ void __launch_bounds__(128) k_train(Weights W, const uint16_t* __restrict__ X,
                                               const uint8_t* __restrict__ Y, long n, long n_total,
                                               float* __restrict__ Gp, float* __restrict__ Lp,
                                               int* __restrict__ err, uint32_t limit) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);
  setup(S);
  const int row = threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float inv_n = 1.0f / float(n_total);
  const long ntiles = (n + 127) / 128;
  uint4 raw = make_uint4(0u, 0u, 0u, 0u);
  uint32_t y = 0;
  auto fetch = [&](long t) {
    const long r = t * 128 + row;
    const bool valid = t < ntiles && r < n;
    raw = valid ? *reinterpret_cast<const uint4*>(X + r * 8) : make_uint4(0u, 0u, 0u, 0u);
    y = valid ? Y[r] : 0u;
  };
  fetch(blockIdx.x);  // before the wait: launched early only behind k_adam, which writes the weights but no rows
  grid_wait();
  grid_release();
  load_weights(S, W);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tbase = S.tmem;
  const uint32_t lane_addr = tbase + (uint32_t(threadIdx.x & ~31) << 16);
  uint32_t phase = 0;
  bool ok = true;
  int tiles_done = 0;
  float gb1 = 0.f, gb2 = 0.f;  // bias gradients of hidden unit `lane`, this warp's rows
  for (long t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++tiles_done) {
    const bool valid = t * 128 + row < n;
    const uint32_t f[3] = {raw.x, raw.y, raw.z}, yb = y;
    *reinterpret_cast<uint4*>(S.x + tc::kmaj(row, 0, 16)) = make_uint4(f[0], f[1], f[2], 0u);
#pragma unroll
    for (int k = 0; k < 6; ++k)
      *reinterpret_cast<uint16_t*>(S.xt + tmaj(k, row)) = uint16_t(f[k / 2] >> (16 * (k & 1)));
    fetch(t + gridDim.x);
    uint32_t pass1, pass2;
    float z3[3];
    ok = forward(S, tbase, phase, &pass1, &pass2, z3, limit);
    if (!ok) break;
    // loss and dZ3
    float dz3[3], l = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float yk = float((yb >> k) & 1u);
      const float z = z3[k];
      const float pk = 1.0f / (1.0f + __expf(-z));
      l += fmaxf(z, 0.f) - z * yk + log1pf(__expf(-fabsf(z)));
      dz3[k] = valid ? (pk - yk) * inv_n : 0.f;
    }
    if (!valid) l = 0.f;
    const uint32_t w01 = pack_bf16(dz3[0], dz3[1]), w2 = pack_bf16(dz3[2], 0.f);
    *reinterpret_cast<uint4*>(S.dz3 + tc::kmaj(row, 0, 16)) = make_uint4(w01, w2, 0u, 0u);
    *reinterpret_cast<uint16_t*>(S.at + tmaj(0, row)) = uint16_t(w01);
    *reinterpret_cast<uint16_t*>(S.at + tmaj(1, row)) = uint16_t(w01 >> 16);
    *reinterpret_cast<uint16_t*>(S.at + tmaj(2, row)) = uint16_t(w2);
    before_issue();
    if (threadIdx.x == 0) {
      tc::fence_after();
      tc::mma_bf16(tbase + C_DH2, desc_k(S.dz3, 16, 0), desc_k(S.w3t, 16, 0), tc::idesc_bf16(128, 32), 0);
      for (int s = 0; s < 8; ++s)
        tc::mma_bf16(tbase + C_GW3, desc_t(S.at, s), desc_t(S.h2t, s), tc::idesc_bf16(128, 32),
                     (tiles_done > 0 || s > 0) ? 1 : 0);
      tc::commit(&S.mbar);
    }
    // while the products run: the loss, and the bias gradients, which sum the same BF16-rounded
    // error terms the matrix products use
    l = warp_sum(l);
    const float g3[3] = {warp_sum(bf_lo(w01)), warp_sum(bf_hi(w01)), warp_sum(bf_lo(w2))};
    if (lane == 0) {
      S.loss[warp] += l;
#pragma unroll
      for (int k = 0; k < 3; ++k) S.gb3[warp][k] += g3[k];
    }
    if (!(ok = wait_mma(S, phase, limit))) break;
    // dZ2
    gb2 += error_train(lane_addr + C_DH2, pass2, S.dz2, S.at, row);
    before_issue();
    if (threadIdx.x == 0) {
      tc::fence_after();
      for (int s = 0; s < 2; ++s)
        tc::mma_bf16(tbase + C_DH1, desc_k(S.dz2, 32, s), desc_k(S.w2t, 32, s), tc::idesc_bf16(128, 32), s);
      for (int s = 0; s < 8; ++s)
        tc::mma_bf16(tbase + C_GW2, desc_t(S.at, s), desc_t(S.h1t, s), tc::idesc_bf16(128, 32),
                     (tiles_done > 0 || s > 0) ? 1 : 0);
      tc::commit(&S.mbar);
    }
    if (!(ok = wait_mma(S, phase, limit))) break;
    // dZ1
    gb1 += error_train(lane_addr + C_DH1, pass1, nullptr, S.at, row);
    before_issue();
    if (threadIdx.x == 0) {
      tc::fence_after();
      for (int s = 0; s < 8; ++s)
        tc::mma_bf16(tbase + C_GW1, desc_t(S.at, s), desc_t(S.xt, s), tc::idesc_bf16(128, 16),
                     (tiles_done > 0 || s > 0) ? 1 : 0);
      tc::commit(&S.mbar);
    }
    if (!(ok = wait_mma(S, phase, limit))) break;
  }
  S.gb1[warp][lane] = gb1;
  S.gb2[warp][lane] = gb2;
  __syncthreads();
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(err, 1);
    // give in-flight MMAs a bounded chance to finish before the columns are released
    tc::mbar_wait(&S.mbar, phase, kWaitLimit);
  }
  // this CTA's partial gradient, every entry of the padded layout written once: rows of the
  // accumulators live in lanes 0..31 (warp 0).  The padded entries are exact zeros (zero input
  // columns 6..15, output rows 3..15); a CTA without a completed tile writes zeros.
  if (threadIdx.x < 32) {
    const bool have = ok && tiles_done > 0;
    float* g = Gp + size_t(blockIdx.x) * kParams;
    float v[16];
    auto put = [&](float* dst, bool keep) {
#pragma unroll
      for (int c = 0; c < 16; c += 4)
        *reinterpret_cast<float4*>(dst + c) =
            keep ? make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    for (int h = 0; h < 2; ++h) {
      if (have) tc::tmem_ld16(lane_addr + C_GW3 + 16 * h, v);
      if (row < 16) put(g + kOffW3 + row * 32 + 16 * h, have && row < 3);
      if (have) tc::tmem_ld16(lane_addr + C_GW2 + 16 * h, v);
      put(g + kOffW2 + row * 32 + 16 * h, have);
    }
    if (have) tc::tmem_ld16(lane_addr + C_GW1, v);
    put(g + kOffW1 + row * 16, have);
    g[kOffB1 + row] = have ? ((S.gb1[0][row] + S.gb1[1][row]) + S.gb1[2][row]) + S.gb1[3][row] : 0.f;
    g[kOffB2 + row] = have ? ((S.gb2[0][row] + S.gb2[1][row]) + S.gb2[2][row]) + S.gb2[3][row] : 0.f;
    if (row < 16)
      g[kOffB3 + row] =
          have && row < 3 ? ((S.gb3[0][row] + S.gb3[1][row]) + S.gb3[2][row]) + S.gb3[3][row] : 0.f;
    if (row == 0) Lp[blockIdx.x] = have ? ((S.loss[0] + S.loss[1]) + S.loss[2]) + S.loss[3] : 0.f;
  }
  teardown(S, tbase);
}

// Probabilities of the three cut-off bits for n rows (rounds of kCRound rows per CTA).
__global__ void __launch_bounds__(128, 4) k_predict(Weights W, const uint16_t* __restrict__ X, long n,
                                                    float* __restrict__ P, int* __restrict__ err,
                                                    uint32_t limit) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SmemC& S = *reinterpret_cast<SmemC*>(smem_raw);
  setup(S, W);
  const uint32_t tbase = S.tmem;
  uint32_t phase = 0;
  bool ok = true;
  const long nround = (n + kCRound - 1) / kCRound;
  for (long rd = blockIdx.x; rd < nround && ok; rd += gridDim.x) {
    const long base = rd * kCRound;
    const int m = int(n - base < kCRound ? n - base : kCRound);
    uint4 in[kCT];
    float z[kCT][3];
#pragma unroll
    for (int t = 0; t < kCT; ++t) {
      const int k = t * 128 + int(threadIdx.x);
      in[t] = k < m ? *reinterpret_cast<const uint4*>(X + (base + k) * 8) : make_uint4(0u, 0u, 0u, 0u);
    }
    ok = forward_rows(S, tbase, phase, in, m, z, limit);
    if (ok)
#pragma unroll
      for (int t = 0; t < kCT; ++t) {
        const int k = t * 128 + int(threadIdx.x);
        if (k < m)
          for (int j = 0; j < 3; ++j) P[(base + k) * 3 + j] = 1.0f / (1.0f + __expf(-z[t][j]));
      }
  }
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(err, 1);
    tc::mbar_wait(&S.mbar, phase, kWaitLimit);
  }
  teardown(S, tbase);
}

// The non-flat stencils of one face of a mixed FV 2D grid, as network rows: the 8 stencils the
// fused stage kernel reconstructs (4 characteristic fields x 2 sides, float, from the double
// state as that kernel sees it), each normalised to [-1, 1] in BF16, with (face << 3 | bit) in
// .w (bit = 2 * field + side).  cq: the 6 cells' conserved values; cp: u, v, H and sqrt|rho| of
// the face's two cells.  Stencils whose six float values are equal are flat and left out: the
// stage kernel takes the linear weights for flat windows by itself.  Returns the bit mask of the
// rows written.
__device__ __forceinline__ uint32_t stencil_rows(float g1, int dir, const float (&cq)[6][4],
                                                 const float (&cp)[2][4], uint32_t face, uint4 (&row)[8]) {
  const Roe2<float> R = roe2<float>(g1, cp[0][3], cp[0][0], cp[0][1], cp[0][2], cp[1][3], cp[1][0],
                                    cp[1][1], cp[1][2]);
  float ch[4][6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    float cc[4];
    roe_left(R, dir, cq[m], cc);
#pragma unroll
    for (int r = 0; r < 4; ++r) ch[r][m] = cc[r];
  }
  uint32_t keep = 0;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const int r = b >> 1, side = b & 1;
    float w[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) w[side ? 5 - m : m] = ch[r][m];
    float mean = 0.f, hi = w[0], lo = w[0];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      mean += w[m];
      hi = fmaxf(hi, w[m]);
      lo = fminf(lo, w[m]);
    }
    row[b] = make_uint4(0u, 0u, 0u, 0u);
    if (hi == lo) continue;
    mean *= (1.0f / 6.0f);
    const float inv = 1.0f / (hi - lo);
    uint32_t f[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const __nv_bfloat16 bv = __float2bfloat16_rn(fminf(1.f, fmaxf(-1.f, (w[m] - mean) * inv)));
      f[m] = *reinterpret_cast<const uint16_t*>(&bv);
    }
    row[b] = make_uint4(f[0] | (f[1] << 16), f[2] | (f[3] << 16), f[4] | (f[5] << 16), face << 3 | uint32_t(b));
    keep |= 1u << b;
  }
  return keep;
}

// Faces per block of the routing pass: A along the sweep direction x B lines across it.
template <int DIR>
struct RouteTile {
  static constexpr int A = DIR == 1 ? 64 : 8, B = DIR == 1 ? 4 : 32;
};

// Learned routing of a mixed FV 2D grid, pass 1 (masks zeroed beforehand), one launch per
// direction: a block stages the float conserved values of its (A + 5) x B cells in shared memory
// (each cell converted once), then one thread per face appends the face's non-flat stencils to
// the row list; appends are aggregated per block, one atomic per block.  A face whose six cells
// are equal has only flat stencils and is skipped before its primitives and eigenvectors.  Rows beyond `cap` are dropped (their stencils keep full TENO).
template <int DIR>
__global__ void __launch_bounds__(256, 6) k_route_prep(Geo G, const double* __restrict__ q, int tiles_a,
                                                    uint4* __restrict__ rows,
                                                    unsigned long long* __restrict__ nrows, long cap,
                                                    const StepState* __restrict__ sst) {
  if (sst && sst->done) return;  // a step after the stop time: no rows (uniform over the block)
  constexpr int A = RouteTile<DIR>::A, B = RouteTile<DIR>::B, L = A + 5, NC = L * B;
  static_assert(A * B == 256, "one face per thread");
  __shared__ float sq[4][NC];  // conserved values, float
  __shared__ int warp_tot[8];
  __shared__ unsigned long long block_base;
  const size_t nc = size_t(G.nx) * G.ny;
  const float g1 = float(G.g1);
  const int n_along = DIR == 1 ? G.nx : G.ny, n_across = DIR == 1 ? G.ny : G.nx;
  const int f0 = int(blockIdx.x % unsigned(tiles_a)) * A, l0 = int(blockIdx.x / unsigned(tiles_a)) * B;
  // staged cell e: along index f0 - 3 + a, line l0 + b; e = b * L + a (x) or a * B + b (y), so
  // that consecutive e are consecutive in memory.  All of a thread's loads are issued before
  // the first conversion.
  constexpr int NS = (NC + 255) / 256;
  double raw[NS][4];
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const int e = int(threadIdx.x) + 256 * j;
    if (e < NC) {
      const int a = DIR == 1 ? e % L : e / B, b = DIR == 1 ? e / L : e % B;
      const int line = min(l0 + b, n_across - 1);  // lines past the grid: their faces are not listed
      const int ia = fused::cmap(f0 - 3 + a, n_along, G.bc);
      const size_t k = DIR == 1 ? size_t(line) * G.nx + ia : size_t(ia) * G.nx + line;
#pragma unroll
      for (int v = 0; v < 4; ++v) raw[j][v] = __ldg(q + v * nc + k);
    }
  }
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    const int e = int(threadIdx.x) + 256 * j;
    if (e < NC)
#pragma unroll
      for (int v = 0; v < 4; ++v) sq[v][e] = fused::d2f(raw[j][v]);
  }
  __syncthreads();
  const int fa = DIR == 1 ? int(threadIdx.x) % A : int(threadIdx.x) / B;
  const int fb = DIR == 1 ? int(threadIdx.x) / A : int(threadIdx.x) % B;
  const int fi = f0 + fa, line = l0 + fb;
  uint4 row[8];
  uint32_t keep = 0;
  if (fi <= n_along && line < n_across) {
    float cq[6][4];
    bool same = true;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      const int e = DIR == 1 ? fb * L + fa + m : (fa + m) * B + fb;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        cq[m][v] = sq[v][e];
        same = same && cq[m][v] == cq[0][v];
      }
    }
    if (!same) {
      float cp[2][4];  // primitives of the face's two cells
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float* c = cq[2 + h];
        // the fused stage kernel's phase-A arithmetic (this unit is also compiled without
        // implicit contraction), so the stencils are the bits that kernel reconstructs
        const float ir = Cst<float>::rcp(c[0]);
        const float u = c[1] * ir, v = c[2] * ir;
        const float p = (c[3] - 0.5f * fmaf(c[2], v, c[1] * u)) * g1;
        cp[h][0] = u;
        cp[h][1] = v;
        cp[h][2] = (c[3] + p) * ir;
        cp[h][3] = Cst<float>::sqrt_(fabsf(c[0]));
      }
      const long nxf = long(G.nx + 1) * G.ny;
      const long face = DIR == 1 ? long(line) * (G.nx + 1) + fi : nxf + long(fi) * G.nx + line;
      keep = stencil_rows(g1, DIR, cq, cp, uint32_t(face), row);
    }
  }
  const int nmine = __popc(keep);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = nmine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_tot[wid] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int tot = 0;
    for (int w = 0; w < 8; ++w) {
      const int t = warp_tot[w];
      warp_tot[w] = tot;
      tot += t;
    }
    block_base = tot ? atomicAdd(nrows, (unsigned long long)tot) : 0ull;
  }
  __syncthreads();
  const unsigned long long base = block_base + warp_tot[wid] + (incl - nmine);
#pragma unroll
  for (int b = 0; b < 8; ++b)
    if (keep >> b & 1u) {
      const unsigned long long slot = base + __popc(keep & ((1u << b) - 1u));
      if (slot < (unsigned long long)cap) rows[slot] = row[b];
    }
}

// Pass 2: the network over the appended rows, in rounds of kCRound rows per CTA; a row whose three
// logits all exceed zthr sets its bit in its face's mask byte.
__global__ void __launch_bounds__(128, 4) k_route_rows(Weights W, const uint4* __restrict__ rows,
                                                       const unsigned long long* __restrict__ nrows,
                                                       long cap, long nxf, uint8_t* __restrict__ mx,
                                                       uint8_t* __restrict__ my, float zthr,
                                                       int* __restrict__ err, uint32_t limit) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  SmemC& S = *reinterpret_cast<SmemC*>(smem_raw);
  const long n = long(min(*nrows, (unsigned long long)cap));
  const long nround = (n + kCRound - 1) / kCRound;
  if (long(blockIdx.x) >= nround) return;  // uniform over the block; no tensor memory taken
  setup(S, W);
  const uint32_t tbase = S.tmem;
  uint32_t phase = 0;
  bool ok = true;
  // this thread's rows of round rd (zero beyond the list)
  auto fetch = [&](long rd, uint4* in) {
    const long base = rd * kCRound;
#pragma unroll
    for (int t = 0; t < kCT; ++t) {
      const long k = base + t * 128 + int(threadIdx.x);
      in[t] = rd < nround && k < n ? rows[k] : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  uint4 in[kCT], next[kCT];
  fetch(blockIdx.x, in);
  for (long rd = blockIdx.x; rd < nround && ok; rd += gridDim.x) {
    const long base = rd * kCRound;
    const int m = int(n - base < kCRound ? n - base : kCRound);
    fetch(rd + gridDim.x, next);  // in flight during this round's products
    float z[kCT][3];
    ok = forward_rows(S, tbase, phase, in, m, z, limit);
    if (ok)
#pragma unroll
      for (int t = 0; t < kCT; ++t) {
        const int k = t * 128 + int(threadIdx.x);
        // the bits of a mask word (4 faces, their rows mostly in neighbouring lanes) meet in the first of
        // its lanes, which writes them, instead of an atomic per row (4096^2, with the packed bias of
        // hidden_row: 2.01 -> 1.55 ms)
        const uint32_t face = in[t].w >> 3, off = face < nxf ? face : face - uint32_t(nxf);
        const bool set = k < m && z[t][0] > zthr && z[t][1] > zthr && z[t][2] > zthr;
        const uint32_t word = (off >> 2) << 1 | (face < nxf ? 0u : 1u);
        uint32_t bits = set ? (1u << (in[t].w & 7u)) << (8 * (off & 3)) : 0u;
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {  // (bits may reach a word's later lanes too: or-ing is idempotent)
          const uint32_t b2 = __shfl_down_sync(0xffffffffu, bits, o), w2 = __shfl_down_sync(0xffffffffu, word, o);
          if (lane + o < 32 && w2 == word) bits |= b2;
        }
        const uint32_t before = __shfl_up_sync(0xffffffffu, word, 1);
        if (bits && (lane == 0 || before != word))
          atomicOr(reinterpret_cast<unsigned int*>(word & 1u ? my : mx) + (word >> 1), bits);
      }
#pragma unroll
    for (int t = 0; t < kCT; ++t) in[t] = next[t];
  }
  if (!ok) {
    if (threadIdx.x == 0) atomicExch(err, 1);
    tc::mbar_wait(&S.mbar, phase, kWaitLimit);
  }
  teardown(S, tbase);
}

// The sum of p[b * stride], b < n, added in order of b, 32 loads in flight.  (Two training epochs of 1e6
// rows: 2.18 ms; with 16 in flight 2.26; with 128 2.80, the longer code being fetched cold at each launch.)
__device__ __forceinline__ float ordered_sum(const float* p, size_t stride, int n) {
  float s = 0.f;
  for (int b = 0; b < n; b += 32) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = b + j < n ? p[size_t(b + j) * stride] : 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (b + j < n) s += v[j];
  }
  return s;
}

// G = the sum of the nblk per-CTA partial gradients, added in CTA order; *loss += the sum of the
// partial losses in CTA order (one thread).  Deterministic for a given grid.
__global__ void k_reduce_grad(const float* __restrict__ Gp, const float* __restrict__ Lp, int nblk,
                              float* __restrict__ G, float* __restrict__ loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kParams) G[i] = ordered_sum(Gp + i, kParams, nblk);
  else if (i == kParams) *loss += ordered_sum(Lp, 1, nblk);
}

// Parameter i's (value p) entries of the device images.
__device__ __forceinline__ void put_images(const Weights& W, int i, float p) {
  __nv_bfloat16* w1 = reinterpret_cast<__nv_bfloat16*>(W.w1);
  __nv_bfloat16* w2 = reinterpret_cast<__nv_bfloat16*>(W.w2);
  __nv_bfloat16* w3 = reinterpret_cast<__nv_bfloat16*>(W.w3);
  __nv_bfloat16* w3t = reinterpret_cast<__nv_bfloat16*>(W.w3t);
  __nv_bfloat16* w2t = reinterpret_cast<__nv_bfloat16*>(W.w2t);
  if (i < kOffB1) {
    w1[i] = __float2bfloat16_rn(i % 16 < 6 ? p : 0.f);
  } else if (i < kOffW2) {
    W.b1[i - kOffB1] = p;
  } else if (i < kOffB2) {
    const int e = i - kOffW2;
    w2[e] = __float2bfloat16_rn(p);
    w2t[(e % 32) * 32 + e / 32] = __float2bfloat16_rn(p);  // W2^T[i][j]
  } else if (i < kOffW3) {
    W.b2[i - kOffB2] = p;
  } else if (i < kOffB3) {
    const int e = i - kOffW3, r = e / 32, k = e % 32;
    w3[e] = __float2bfloat16_rn(r < 3 ? p : 0.f);
    w3t[k * 16 + r] = __float2bfloat16_rn(r < 3 ? p : 0.f);  // W3^T[j][k]
  } else {
    W.b3[i - kOffB3] = i - kOffB3 < 3 ? p : 0.f;
  }
}
__global__ void k_images(const float* __restrict__ P, Weights W) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kParams) put_images(W, i, P[i]);
}

// After k_train, one thread per parameter: the gradient (the partials added in CTA order, as
// k_reduce_grad), Adam on the FP32 master parameters (padded layout) and the images of the new value;
// one thread more for the loss.  Bound by latency (34 blocks of 64 threads, the partials from L2, 32 loads
// in flight each).  Alone from cold caches the three kernels that did this took 9.9 + 4 + 4 us, this one 11.
__global__ void __launch_bounds__(64) k_adam(const float* __restrict__ Gp, const float* __restrict__ Lp, int nblk,
                                             float* __restrict__ P, float* __restrict__ M, float* __restrict__ V,
                                             float* __restrict__ loss, Weights W, float lr, float b1, float b2,
                                             float eps, int t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  grid_wait();
  grid_release();
  Gp = after_wait(Gp);
  Lp = after_wait(Lp);
  P = after_wait(P);
  M = after_wait(M);
  V = after_wait(V);
  loss = after_wait(loss);
  if (i == kParams) *loss += ordered_sum(Lp, 1, nblk);
  if (i >= kParams) return;
  const float m0 = M[i], v0 = V[i], p0 = P[i];
  const float g = ordered_sum(Gp + i, kParams, nblk);
  const float m = b1 * m0 + (1.f - b1) * g;
  const float v = b2 * v0 + (1.f - b2) * g * g;
  M[i] = m;
  V[i] = v;
  const float mh = m / (1.f - powf(b1, float(t))), vh = v / (1.f - powf(b2, float(t)));
  const float p = p0 - lr * mh / (sqrtf(vh) + eps);
  P[i] = p;
  put_images(W, i, p);
}

// Converts float rows [n][6] to the bf16 training layout [n][8].
__global__ void k_pack_inputs(const float* __restrict__ in, uint16_t* __restrict__ out, long n) {
  const long r = blockIdx.x * long(blockDim.x) + threadIdx.x;
  if (r >= n) return;
  for (int k = 0; k < 8; ++k) {
    const __nv_bfloat16 b = __float2bfloat16_rn(k < 6 ? in[r * 6 + k] : 0.f);
    out[r * 8 + k] = *reinterpret_cast<const uint16_t*>(&b);
  }
}

}  // namespace

size_t smem_bytes() { return sizeof(Smem); }

}  // namespace mlp
}  // namespace hteno

using namespace hteno;
using namespace hteno::mlp;

struct hteno_mlp {
  Weights W{};          // device images
  float* P = nullptr;   // FP32 master parameters (padded)
  float* G = nullptr;   // gradient (padded), the ordered sum of the per-CTA partials
  float* Gp = nullptr;  // per-CTA partial gradients [2 * sms][kParams] and partial losses
  float* Lp = nullptr;
  float* M = nullptr;   // Adam moments
  float* V = nullptr;
  float* loss = nullptr;
  int* err = nullptr;
  void* img = nullptr;  // backing store of W
  int t = 0;            // Adam step
  uint32_t wait_limit = kWaitLimit;  // polls of a tensor-core completion wait
  int sms = 148;
  cudaStream_t stream = nullptr;
  std::string msg;
};

namespace {

int merr(hteno_mlp* m, cudaError_t e, const char* what) {
  if (e == cudaSuccess) return HTENO_OK;
  m->msg = std::string(what) + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? HTENO_ERR_OOM : HTENO_ERR_CUDA;
}

int set_attr() {
  static int done = 0;
  if (done) return HTENO_OK;
  const int sm = int(mlp::smem_bytes());
  const int smc = int(mlp::kSmemCBytes);
  if (cudaFuncSetAttribute(k_train, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) != cudaSuccess ||
      cudaFuncSetAttribute(k_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, smc) != cudaSuccess ||
      cudaFuncSetAttribute(k_route_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, smc) != cudaSuccess)
    return HTENO_ERR_CUDA;
  done = 1;
  return HTENO_OK;
}

int check_err(hteno_mlp* m) {
  int h = 0;
  cudaError_t e = cudaMemcpyAsync(&h, m->err, sizeof(int), cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) return merr(m, e, "mlp");
  if (h) {
    m->msg = "tensor-core wait timed out";
    cudaMemsetAsync(m->err, 0, sizeof(int), m->stream);
    return HTENO_ERR_TIMEOUT;
  }
  return HTENO_OK;
}

// compact public layout <-> padded internal layout
void to_padded(const float* c, float* p) {
  std::memset(p, 0, kParams * sizeof(float));
  for (int j = 0; j < 32; ++j)
    for (int i = 0; i < 6; ++i) p[kOffW1 + j * 16 + i] = c[j * 6 + i];
  for (int j = 0; j < 32; ++j) p[kOffB1 + j] = c[192 + j];
  for (int e = 0; e < 1024; ++e) p[kOffW2 + e] = c[224 + e];
  for (int j = 0; j < 32; ++j) p[kOffB2 + j] = c[1248 + j];
  for (int e = 0; e < 96; ++e) p[kOffW3 + e] = c[1280 + e];
  for (int k = 0; k < 3; ++k) p[kOffB3 + k] = c[1376 + k];
}
void from_padded(const float* p, float* c) {
  for (int j = 0; j < 32; ++j)
    for (int i = 0; i < 6; ++i) c[j * 6 + i] = p[kOffW1 + j * 16 + i];
  for (int j = 0; j < 32; ++j) c[192 + j] = p[kOffB1 + j];
  for (int e = 0; e < 1024; ++e) c[224 + e] = p[kOffW2 + e];
  for (int j = 0; j < 32; ++j) c[1248 + j] = p[kOffB2 + j];
  for (int e = 0; e < 96; ++e) c[1280 + e] = p[kOffW3 + e];
  for (int k = 0; k < 3; ++k) c[1376 + k] = p[kOffB3 + k];
}

int refresh_images(hteno_mlp* m) {
  k_images<<<(kParams + 255) / 256, 256, 0, m->stream>>>(m->P, m->W);
  return merr(m, cudaGetLastError(), "weight images");
}

}  // namespace

namespace hteno {

// Route masks of a mixed FV 2D grid from its current state: the masks are zeroed, k_route_prep
// (x faces, then y faces) lists the non-flat stencils (at most `cap` rows, scratch owned by the caller), k_route_rows runs
// the network on them.  *nrows receives the number of non-flat stencils.
int mlp_classify(hteno_mlp* m, const Geo& G, const double* q, uint8_t* mx, uint8_t* my, float thr,
                 uint4* rows, unsigned long long* nrows, long cap, cudaStream_t st,
                 const StepState* sst) {
  const long nxf = long(G.nx + 1) * G.ny, nyf = long(G.ny + 1) * G.nx;
  cudaMemsetAsync(mx, 0, size_t(nxf), st);
  cudaMemsetAsync(my, 0, size_t(nyf), st);
  cudaMemsetAsync(nrows, 0, sizeof(unsigned long long), st);
  {
    using T1 = RouteTile<1>;
    using T2 = RouteTile<2>;
    const int ta1 = (G.nx + 1 + T1::A - 1) / T1::A, tb1 = (G.ny + T1::B - 1) / T1::B;
    const int ta2 = (G.ny + 1 + T2::A - 1) / T2::A, tb2 = (G.nx + T2::B - 1) / T2::B;
    k_route_prep<1><<<unsigned(ta1) * unsigned(tb1), 256, 0, st>>>(G, q, ta1, rows, nrows, cap, sst);
    k_route_prep<2><<<unsigned(ta2) * unsigned(tb2), 256, 0, st>>>(G, q, ta2, rows, nrows, cap, sst);
  }
  const float zthr = std::log(thr / (1.0f - thr));  // sigmoid(z) > thr  <=>  z > logit(thr)
  k_route_rows<<<4 * m->sms, 128, mlp::kSmemCBytes, st>>>(m->W, rows, nrows, cap, nxf, mx, my, zthr,
                                                          m->err, m->wait_limit);
  return cudaGetLastError() == cudaSuccess ? HTENO_OK : HTENO_ERR_CUDA;
}

int mlp_status(hteno_mlp* m, cudaStream_t st) {
  int h = 0;
  if (cudaMemcpyAsync(&h, m->err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return HTENO_ERR_CUDA;
  return h ? HTENO_ERR_TIMEOUT : HTENO_OK;
}

}  // namespace hteno

extern "C" {

int hteno_mlp_create(unsigned long long seed, hteno_mlp** out) {
  if (!out) return HTENO_ERR_INVALID_ARG;
  *out = nullptr;
  hteno_mlp* m = new (std::nothrow) hteno_mlp();
  if (!m) return HTENO_ERR_OOM;
  auto fail = [&](int code) {
    cudaFree(m->P); cudaFree(m->G); cudaFree(m->M); cudaFree(m->V); cudaFree(m->loss);
    cudaFree(m->err); cudaFree(m->img); cudaFree(m->Gp); cudaFree(m->Lp);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return code;
  };
  if (set_attr() != HTENO_OK) return fail(HTENO_ERR_CUDA);
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(HTENO_ERR_CUDA);
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t pb = kParams * sizeof(float);
  if (cudaMalloc(&m->P, pb) || cudaMalloc(&m->G, pb) || cudaMalloc(&m->M, pb) || cudaMalloc(&m->V, pb) ||
      cudaMalloc(&m->loss, sizeof(float)) || cudaMalloc(&m->err, sizeof(int)) ||
      cudaMalloc(&m->img, kImageBytes) || cudaMalloc(&m->Gp, 2 * size_t(m->sms) * pb) ||
      cudaMalloc(&m->Lp, 2 * size_t(m->sms) * sizeof(float)))
    return fail(HTENO_ERR_OOM);
  char* b = static_cast<char*>(m->img);
  m->W.w1 = b; m->W.w2 = b + 1024; m->W.w3 = b + 3072; m->W.w3t = b + 4096; m->W.w2t = b + 5120;
  m->W.b1 = reinterpret_cast<float*>(b + 7168);
  m->W.b2 = m->W.b1 + 32;
  m->W.b3 = m->W.b2 + 32;
  // He-uniform initialisation of the weights, zero biases
  std::mt19937_64 rng(seed);
  std::vector<float> c(kPublicParams, 0.f), p(kParams);
  auto uni = [&](float a) { return float((double(rng() >> 11) * 0x1.0p-53 * 2.0 - 1.0) * a); };
  for (int e = 0; e < 192; ++e) c[e] = uni(std::sqrt(6.f / 6.f));
  for (int e = 0; e < 1024; ++e) c[224 + e] = uni(std::sqrt(6.f / 32.f));
  for (int e = 0; e < 96; ++e) c[1280 + e] = uni(std::sqrt(6.f / 32.f));
  to_padded(c.data(), p.data());
  if (cudaMemcpy(m->P, p.data(), pb, cudaMemcpyHostToDevice) || cudaMemset(m->G, 0, pb) ||
      cudaMemset(m->M, 0, pb) || cudaMemset(m->V, 0, pb) || cudaMemset(m->err, 0, sizeof(int)) ||
      cudaMemset(m->img, 0, kImageBytes))
    return fail(HTENO_ERR_CUDA);
  if (refresh_images(m) != HTENO_OK || cudaStreamSynchronize(m->stream) != cudaSuccess)
    return fail(HTENO_ERR_CUDA);
  *out = m;
  return HTENO_OK;
}

int hteno_mlp_destroy(hteno_mlp* m) {
  if (!m) return HTENO_ERR_INVALID_ARG;
  cudaStreamSynchronize(m->stream);
  cudaFree(m->P); cudaFree(m->G); cudaFree(m->M); cudaFree(m->V); cudaFree(m->loss);
  cudaFree(m->err); cudaFree(m->img); cudaFree(m->Gp); cudaFree(m->Lp);
  cudaStreamDestroy(m->stream);
  delete m;
  return HTENO_OK;
}

int hteno_mlp_num_params(void) { return kPublicParams; }

int hteno_mlp_set_params(hteno_mlp* m, const float* params) {
  if (!m || !params) return HTENO_ERR_INVALID_ARG;
  std::vector<float> p(kParams);
  to_padded(params, p.data());
  cudaError_t e = cudaMemcpyAsync(m->P, p.data(), kParams * sizeof(float), cudaMemcpyHostToDevice, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) return merr(m, e, "set params");
  m->t = 0;
  cudaMemsetAsync(m->M, 0, kParams * sizeof(float), m->stream);
  cudaMemsetAsync(m->V, 0, kParams * sizeof(float), m->stream);
  const int rc = refresh_images(m);
  return rc ? rc : merr(m, cudaStreamSynchronize(m->stream), "set params");
}

int hteno_mlp_get_params(hteno_mlp* m, float* params) {
  if (!m || !params) return HTENO_ERR_INVALID_ARG;
  std::vector<float> p(kParams);
  cudaError_t e = cudaMemcpyAsync(p.data(), m->P, kParams * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) return merr(m, e, "get params");
  from_padded(p.data(), params);
  return HTENO_OK;
}

// Gradient of the mean BCE loss over n rows (x: device bf16 [n][8], y: device u8 [n]); grads in
// the public layout (host), *loss = mean loss.
int hteno_mlp_grad(hteno_mlp* m, const uint16_t* x, const uint8_t* y, long n, float* grads, float* loss) {
  if (!m || !x || !y || n <= 0 || !grads) return HTENO_ERR_INVALID_ARG;
  cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream);
  const long tiles = (n + 127) / 128;
  const int grid = int(std::min<long>(tiles, 2L * m->sms));
  k_train<<<grid, 128, mlp::smem_bytes(), m->stream>>>(m->W, x, y, n, n, m->Gp, m->Lp, m->err,
                                                       m->wait_limit);
  k_reduce_grad<<<(kParams + 256) / 256, 256, 0, m->stream>>>(m->Gp, m->Lp, grid, m->G, m->loss);
  int rc = merr(m, cudaGetLastError(), "k_train");
  if (rc) return rc;
  rc = check_err(m);
  if (rc) return rc;
  std::vector<float> g(kParams);
  float l = 0.f;
  cudaError_t e = cudaMemcpyAsync(g.data(), m->G, kParams * sizeof(float), cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) return merr(m, e, "grad copy");
  from_padded(g.data(), grads);
  if (loss) *loss = l / float(n);
  return HTENO_OK;
}

// Mini-batch Adam over the n rows for `epochs` passes (batches are contiguous slices; shuffle the
// data beforehand).  *loss receives the mean loss of the last epoch.
int hteno_mlp_train(hteno_mlp* m, const uint16_t* x, const uint8_t* y, long n, int epochs, long batch,
                    float lr, float* loss) {
  if (!m || !x || !y || n <= 0 || epochs < 0 || batch <= 0 || !(lr > 0.f)) return HTENO_ERR_INVALID_ARG;
  float last = 0.f;
  for (int ep = 0; ep < epochs; ++ep) {
    cudaMemsetAsync(m->loss, 0, sizeof(float), m->stream);
    for (long off = 0; off < n; off += batch) {
      const long nb = std::min(batch, n - off);
      const long tiles = (nb + 127) / 128;
      const int grid = int(std::min<long>(tiles, 2L * m->sms));
      ++m->t;
      // an epoch's first batch waits for whatever is before it: k_train reads rows before its grid_wait,
      // and the kernel before it may be the one that wrote them; the later batches follow k_adam
      cudaError_t e = launch_early(off > 0, k_train, grid, 128, mlp::smem_bytes(), m->stream, m->W, x + off * 8, y + off, nb,
                                   nb, m->Gp, m->Lp, m->err, m->wait_limit);
      if (e == cudaSuccess)
        e = launch_early(true, k_adam, (kParams + 64) / 64, 64, 0, m->stream, m->Gp, m->Lp, grid, m->P, m->M, m->V,
                         m->loss, m->W, lr, 0.9f, 0.999f, 1e-8f, m->t);
      if (e != cudaSuccess) return merr(m, e, "train launch");
    }
    int rc = merr(m, cudaGetLastError(), "train launch");
    if (rc) return rc;
    rc = check_err(m);
    if (rc) return rc;
    float l = 0.f;
    cudaMemcpy(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost);
    last = l / float(n);
  }
  if (loss) *loss = last;
  return HTENO_OK;
}

// Probabilities of the three cut-off bits: x device bf16 [n][8] -> p device float [n][3].
int hteno_mlp_predict(hteno_mlp* m, const uint16_t* x, long n, float* p) {
  if (!m || !x || n <= 0 || !p) return HTENO_ERR_INVALID_ARG;
  const long rounds = (n + mlp::kCRound - 1) / mlp::kCRound;
  const int grid = int(std::min<long>(rounds, 4L * m->sms));
  k_predict<<<grid, 128, mlp::kSmemCBytes, m->stream>>>(m->W, x, n, p, m->err, m->wait_limit);
  const int rc = merr(m, cudaGetLastError(), "k_predict");
  return rc ? rc : check_err(m);
}

// float [n][6] (device) -> bf16 training rows [n][8] (device).
int hteno_mlp_pack(hteno_mlp* m, const float* in, uint16_t* out, long n) {
  if (!m || !in || !out || n <= 0) return HTENO_ERR_INVALID_ARG;
  k_pack_inputs<<<unsigned((n + 255) / 256), 256, 0, m->stream>>>(in, out, n);
  const int rc = merr(m, cudaGetLastError(), "pack");
  return rc ? rc : merr(m, cudaStreamSynchronize(m->stream), "pack");
}

int hteno_mlp_set_wait_limit(hteno_mlp* m, unsigned int polls) {
  if (!m) return HTENO_ERR_INVALID_ARG;
  m->wait_limit = polls;
  return HTENO_OK;
}

const char* hteno_mlp_last_error(hteno_mlp* m) { return m ? m->msg.c_str() : "null handle"; }

}  // extern "C"
