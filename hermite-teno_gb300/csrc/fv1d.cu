// FV::System1D on the GPU (FV_System1D.cpp:158-292): characteristic reconstruction (teno5,
// teno5i as shipped, or linear) from a 6-cell stencil, HLLC or characteristic Rusanov, SSP-RK3.
// A 1D grid of a few hundred cells is a latency case: in double a step is three launches, one per
// stage (k1_stage); in mixed precision 2 + 3 x 2 small ones with one thread per face / per cell.  The
// host replays them without synchronising (dt on the device).  In double the bit-reproducible
// functions (parity_math.cuh) are used; compiled with --fmad=false.
#include <type_traits>

#include "hteno_internal.h"
#include "parity_math.cuh"
#include "harvest.cuh"

namespace hteno {
namespace {

__constant__ DevConst c_dev;
__device__ DevConst g_dev;  // the same in global memory (double: par::ldk)
unsigned long long g_mask = 0;
std::mutex g_mu;

#include "common_kernels.cuh"

constexpr int kThreads = 64;

struct Geo1 {
  int nx, bc, recon, flux;
  double dx, area, rarea, gamma, g1;  // rarea = 1 / area
};

// calcPrimitiveVariable (FV_System1D.cpp:95-119); the divisions share d, the density
__device__ __forceinline__ void cell_prim1(double g1, const double* q, const par::Den& d, par::fp* w, par::fp& h,
                                           par::fp& sr) {
  const par::fp qf[3] = {q[0], q[1], q[2]};
  par::primitive1(g1, qf, d, w);
  h = par::quot(qf[2] + w[2], d);
  sr = par::sqrt_abs(w[0]);
}
__device__ __forceinline__ void cell_prim1(double g1, const double* q, double* w, double& h, double& sr) {
  par::fp wf[3], hf, sf;
  cell_prim1(g1, q, par::den_of(q[0]), wf, hf, sf);
  for (int k = 0; k < 3; ++k) w[k] = wf[k].v;
  h = hf.v;
  sr = sf.v;
}

// The max wave speed of a new state and, for the stages in double, its cells' u, h, sqrt|rho|
// (prim [3][nx]; null in mixed precision).
__global__ void k1_init(Geo1 G, const double* __restrict__ q, double* __restrict__ prim, StepState* st) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ms = 0.0;
  if (i < G.nx) {
    const double qq[3] = {q[i], q[G.nx + i], q[2 * G.nx + i]};
    const par::Den d = par::den_of(qq[0]);
    par::fp w[3], h, sr;
    cell_prim1(G.g1, qq, d, w, h, sr);
    if (prim) {
      prim[i] = w[1].v;
      prim[G.nx + i] = h.v;
      prim[2 * G.nx + i] = sr.v;
    }
    ms = par::max_speed1(G.gamma, w[1], w[2], d);
  }
  block_max_to(ms, &st->maxbits);
}

// face f in [0, nx] between cells f-1 and f (FV_System1D.cpp:194-235), mixed precision
__global__ void __launch_bounds__(kThreads) k1_flux_f(Geo1 G, const double* __restrict__ q,
                                                      float* __restrict__ F, const StepState* st) {
  if (st->done) return;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f > G.nx) return;
  const int n = G.nx;
  double qa[3], qb[3], wa[3], wb[3], ha, hb, sa, sb;
  const int ca = bmap(f - 1, n, G.bc), cb = bmap(f, n, G.bc);
  for (int v = 0; v < 3; ++v) {
    qa[v] = q[v * n + ca];
    qb[v] = q[v * n + cb];
  }
  cell_prim1(G.g1, qa, wa, ha, sa);
  cell_prim1(G.g1, qb, wb, hb, sb);
  float Ff[3];
  const Roe1<float> R = roe1<float>(float(G.g1), float(sa), float(wa[1]), float(ha), float(sb), float(wb[1]), float(hb));
  float ch[3][6];
  for (int m = 0; m < 6; ++m) {
    const int c = bmap(f - 3 + m, n, G.bc);
    float qq[3] = {float(q[c]), float(q[n + c]), float(q[2 * n + c])}, cc[3];
    roe1_left(R, qq, cc);
    for (int r = 0; r < 3; ++r) ch[r][m] = cc[r];
  }
  float cl[3], cr[3], ql[3], qr[3];
  for (int r = 0; r < 3; ++r) lagrange_recon(c_dev, G.recon, ch[r], cl[r], cr[r]);
  roe1_right(R, cl, ql);
  roe1_right(R, cr, qr);
  if (G.flux == HTENO_FLUX_HLLC) hllc1(float(G.g1), ql, qr, Ff);
  else rusanov1(float(G.gamma), float(G.g1), R, ql, qr, Ff);
  for (int v = 0; v < 3; ++v) F[v * (n + 1) + f] = Ff[v];
}

// One stage of a step in double, one launch: a block computes the fluxes of FB consecutive faces and
// updates the FB - 1 cells between them.  8 lanes per face: lane r + 4 s (r < 3 the characteristic
// field, s the side) projects its field's 6-cell stencil and reconstructs one side; then every lane
// of a side projects that side back and computes its part of the flux, and the two sides meet by
// shuffles.  Then 4 lanes per cell, one per conserved variable, take the SSP-RK3 stage and, together,
// the new state's primitives.
//
// An FP64 unit takes 64 cycles per warp instruction however many lanes are active, and a grid of a
// few hundred cells gives each of the chip's 608 less than a warp: the time is the number of FP64
// operations in sequence, so the lanes share a face's work, a cell's primitives are computed once
// and kept, and edge faces are computed by both blocks they border.  FB = 4 (one warp per block)
// spreads 456 cells over one warp per SM.  400 cells: 98 -> 53 us a step (eight launches before).
//
// The stage reads the state and primitives of `qin`, `pin` with its neighbours and the step-start
// state `qbase` cell by cell, and writes `qout`, `pout`: no block reads what another writes.  Stage 1
// also starts the step (timeStepping, :274-292): every block finds dt or the stop from the same
// values, one records them; stage 2 resets the wave speed that stage 3 collects; stage 3 advances t.
template <int FB>
__global__ void __launch_bounds__(8 * FB) k1_stage(Geo1 G, int stage, const double* __restrict__ qin,
                                                   const double* __restrict__ pin, const double* qbase,
                                                   double* qout, double* __restrict__ pout, StepState* st) {
  using par::fp;
  __shared__ double sF[3][FB];
  const bool first = blockIdx.x == 0 && threadIdx.x == 0;
  double dt;
  if (stage == 1) {
    if (st->done || !(st->t < st->t_final)) {
      if (first) st->done = 1;
      return;
    }
    dt = st->dt_scale / __longlong_as_double(static_cast<long long>(st->maxbits));
    dt = st->t + dt > st->t_final ? st->t_final - st->t : dt;
    if (first) st->dt = dt;
  } else {
    if (st->done) return;
    dt = st->dt;
    if (first && stage == 2) st->maxbits = 0ull;
    if (first && stage == 3) {
      st->t += dt;
      st->steps += 1;
    }
  }
  const int n = G.nx, tid = threadIdx.x;
  const int c0 = blockIdx.x * (FB - 1), f = min(c0 + (tid >> 3), n);  // faces past the last compute it again
  const int l = tid & 7, r = l & 3, side = l >> 2;
  const int ca = bmap(f - 1, n, G.bc), cb = bmap(f, n, G.bc);
  fp R[9], L[9];
  par::eig1(G.g1, pin[2 * n + ca], pin[ca], pin[n + ca], pin[2 * n + cb], pin[cb], pin[n + cb], R, L);
  const fp l0 = r == 0 ? L[0] : r == 1 ? L[3] : L[6];
  const fp l1 = r == 0 ? L[1] : r == 1 ? L[4] : L[7];
  const fp l2 = r == 0 ? L[2] : r == 1 ? L[5] : L[8];
  double ch[6];
#pragma unroll
  for (int m = 0; m < 6; ++m) {
    const int c = bmap(f - 3 + m, n, G.bc);
    const fp qq[3] = {qin[c], qin[n + c], qin[2 * n + c]};
    ch[m] = par::dot3(l0, l1, l2, qq).v;  // row r of par::mv3
  }
  const double val = par::lagrange_side(g_dev, G.recon, ch, side);  // lanes r = 3 repeat r = 2
  const int base = tid & 24;
  fp c3[3], qs[3], F[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) c3[k] = __shfl_sync(0xffffffffu, val, base + 4 * side + k);
  par::mv3(R, c3, qs);  // transformToConservative (FV_System1D.h:48-51)
  if (G.flux == HTENO_FLUX_HLLC) {
    const par::Den rho = par::den_of(qs[0]);
    const par::Hllc1Side own = par::hllc1_side(G.g1, qs, rho);
    auto swap = [&](fp x) { return fp(__shfl_xor_sync(0xffffffffu, x.v, 4)); };
    par::Hllc1Side other;
#pragma unroll
    for (int k = 0; k < 3; ++k) other.q[k] = swap(own.q[k]);
    other.w[0] = other.q[0];
    other.w[1] = swap(own.w[1]);
    other.w[2] = swap(own.w[2]);
    other.h = swap(own.h);
    other.c = swap(own.c);
    par::Den rl = rho;  // the left density, in the lanes of both sides
    const fp oy = swap(rho.y);
    if (side) rl = par::Den{other.q[0], oy, par::mid_range(other.q[0].v)};
    par::Hllc1Side lt = own, rt = other;
    if (side) {
      lt = other;
      rt = own;
    }
    par::hllc1(G.g1, lt, rt, rl, F);
  } else {
    fp ql[3], qr[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const fp x = __shfl_xor_sync(0xffffffffu, qs[k].v, 4);
      ql[k] = side ? x : qs[k];
      qr[k] = side ? qs[k] : x;
    }
    par::rusanov1(par::sides1_of(G.gamma, G.g1, ql, qr), L, R, ql, qr, F);
  }
  if (l < 3) sF[l][tid >> 3] = (l == 0 ? F[0] : l == 1 ? F[1] : F[2]).v;
  __syncthreads();
  // rhs (:237-240) + RungeKutta3 (:243-272): cell c0 + (tid >> 2), variable tid & 3
  const int j = tid >> 2, v = min(tid & 3, 2), jj = min(j, FB - 2), i = min(c0 + jj, n - 1);
  const bool mine = j < FB - 1 && c0 + j < n;
  const par::Den area{G.area, G.rarea, par::mid_range(G.area)};
  const fp rhs = par::quot(fp(sF[v][jj]) - sF[v][jj + 1], area);
  const double cur = qin[v * n + i];
  const double qn = par::rk3(stage == 1 ? cur : qbase[v * n + i], cur, rhs, dt, stage);
  double q3[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) q3[k] = __shfl_sync(0xffffffffu, qn, (tid & 28) + k);
  const par::Den d = par::den_of(q3[0]);
  fp w[3], h, sr;
  cell_prim1(G.g1, q3, d, w, h, sr);
  if (mine && (tid & 3) < 3) {
    qout[v * n + i] = qn;
    pout[v * n + i] = (v == 0 ? w[1] : v == 1 ? h : sr).v;
  }
  if (mine && (tid & 3) == 0) {
    int bad = par::nan_bits(q3[0]) || par::nan_bits(q3[1]) || par::nan_bits(q3[2]) ? 1 : 0;
    bad |= par::nonpositive_bits(q3[0]) || par::nonpositive_bits(w[2].v) ? 2 : 0;
    if (bad) atomicOr(&st->status, bad);
  }
  if (stage == 3) block_max_to(mine ? par::max_speed1(G.gamma, w[1], w[2], d) : 0.0, &st->maxbits);
}

// rhs (FV_System1D.cpp:237-240) + RungeKutta3 (:243-272); max wave speed on the last stage; mixed
// precision
__global__ void k1_update_f(Geo1 G, int stage, const float* __restrict__ F, double* __restrict__ q,
                            double* __restrict__ q0, StepState* st) {
  if (st->done) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = G.nx;
  double ms = 0.0;
  int bad = 0;
  if (i < n) {
    const double dt = st->dt;
    double qn[3];
    for (int v = 0; v < 3; ++v) {
      const double rhs = (double(F[v * (n + 1) + i]) - double(F[v * (n + 1) + i + 1])) / G.area;
      const double cur = q[v * n + i];
      double base;
      if (stage == 1) {
        q0[v * n + i] = cur;
        base = cur;
      } else {
        base = q0[v * n + i];
      }
      qn[v] = par::rk3(base, cur, rhs, dt, stage);
      q[v * n + i] = qn[v];
    }
    const par::Den d = par::den_of(qn[0]);
    par::fp w[3], h, sr;
    cell_prim1(G.g1, qn, d, w, h, sr);
    if (stage == 3) ms = par::max_speed1(G.gamma, w[1], w[2], d);
    bad = (isnan(qn[0]) || isnan(qn[1]) || isnan(qn[2])) ? 1 : 0;
    bad |= (qn[0] <= 0.0 || w[2].v <= 0.0) ? 2 : 0;
  }
  if (stage == 3) block_max_to(ms, &st->maxbits);
  if (bad) atomicOr(&st->status, bad);
}

// Training stencils of the learned classifier (harvest.cuh): every face, 3 characteristic
// fields, both sides, each kept with probability p.
__global__ void __launch_bounds__(kThreads) k1_harvest(Geo1 G, const double* __restrict__ q, double p,
                                                       unsigned long long seed, uint16_t* X, uint8_t* Y,
                                                       long cap, unsigned long long* count) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f > G.nx) return;
  const int n = G.nx;
  double qa[3], qb[3], wa[3], wb[3], ha, hb, sa, sb;
  const int ca = bmap(f - 1, n, G.bc), cb = bmap(f, n, G.bc);
  for (int v = 0; v < 3; ++v) {
    qa[v] = q[v * n + ca];
    qb[v] = q[v * n + cb];
  }
  cell_prim1(G.g1, qa, wa, ha, sa);
  cell_prim1(G.g1, qb, wb, hb, sb);
  par::fp R[9], L[9];
  double ch[3][6];
  par::eig1(G.g1, sa, wa[1], ha, sb, wb[1], hb, R, L);
  for (int m = 0; m < 6; ++m) {
    const int c = bmap(f - 3 + m, n, G.bc);
    const par::fp qq[3] = {q[c], q[n + c], q[2 * n + c]};
    par::fp cc[3];
    par::mv3(L, qq, cc);
    for (int r = 0; r < 3; ++r) ch[r][m] = cc[r].v;
  }
  for (int r = 0; r < 3; ++r)
    harvest::emit_both(ch[r], G.recon == HTENO_RECON_TENO5I, seed, (uint64_t(r) << 40) + uint64_t(f),
                       p, X, Y, cap, count);
}

// KXRCF troubled-cell sensor of FV::System1D::rhs (FV_System1D.cpp:166-192): from the density
// averages, the two one-sided face values of the upwind face (chosen by the sign of rho*u),
// flagged when |h1 - h2| / ((dx/2)^1.5 |rho_i|) > 1.  The reference computes the flag for cells
// s+1 .. nxx-s-2 of its ghost-padded array (every interior cell) and reconstructs with teno5i
// either way; here the flags are an output.
__global__ void k1_kxrcf(Geo1 G, const double* __restrict__ q, double crm, uint8_t* __restrict__ flag) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= G.nx) return;
  const int n = G.nx;
  auto rho = [&](int k) { return q[bmap(k, n, G.bc)]; };
  double h1, h2;
  if (q[n + i] < 0.0) {
    h1 = (2.0 * rho(i - 1) + 5.0 * rho(i) - rho(i + 1)) / 6.0;
    h2 = (-rho(i - 2) + 5.0 * rho(i - 1) + 2.0 * rho(i)) / 6.0;
  } else {
    h2 = (2.0 * rho(i) + 5.0 * rho(i + 1) - rho(i + 2)) / 6.0;
    h1 = (-rho(i - 1) + 5.0 * rho(i) + 2.0 * rho(i + 1)) / 6.0;
  }
  flag[i] = fabs(h1 - h2) / (crm * fabs(rho(i))) > 1.0 ? 1 : 0;
}

Geo1 geo1_of(const hteno_solver* s) {
  Geo1 G;
  G.nx = s->cfg.nx;
  G.bc = s->cfg.bc;
  G.recon = s->cfg.recon;
  G.flux = s->cfg.flux;
  G.dx = s->dx;
  G.area = s->dx;
  G.rarea = 1.0 / s->dx;
  G.gamma = s->cfg.gamma;
  G.g1 = s->cfg.gamma - 1.0;
  return G;
}

// Work buffer in double: the state between stages 2 and 3 [3][nx] and the primitives of the three
// stage inputs [3][3][nx] (the state between stages 1 and 2 is q0); in mixed precision the face
// fluxes [3][nx + 1].
constexpr int kWorkArrays = 12;

template <int FB>
void launch_stages(hteno_solver* s, const Geo1& G, cudaStream_t cs) {
  const unsigned grid = unsigned((G.nx + FB - 2) / (FB - 1));
  double* w = static_cast<double*>(s->work);
  const size_t m = 3 * size_t(G.nx);
  k1_stage<FB><<<grid, 8 * FB, 0, cs>>>(G, 1, s->q, w + m, s->q, s->q0, w + 2 * m, s->dstate);
  k1_stage<FB><<<grid, 8 * FB, 0, cs>>>(G, 2, s->q0, w + 2 * m, s->q, w, w + 3 * m, s->dstate);
  k1_stage<FB><<<grid, 8 * FB, 0, cs>>>(G, 3, w, w + 3 * m, s->q, s->q, w + m, s->dstate);
}

void launch_step(hteno_solver* s, const Geo1& G, cudaStream_t cs) {
  if (s->cfg.precision == HTENO_PREC_FP64) {
    // 4 faces a block (a third of them computed twice) while that is at most a warp per SM
    // sub-partition; then 16 (a fifteenth).  32 steps, 4 / 16 faces, HLLC and Rusanov: 400 cells 1.75 / 1.82 ms (HLLC),
    // 1824 1.80 / 1.84, 1.63 / 1.63; 2000 1.97 / 1.83, 1.72 / 1.55; 2400 2.23 / 2.47, 1.90 / 2.30; 3500 2.77 / 2.76,
    // 2.43 / 2.43; 5000 3.68 / 3.86, 3.27 / 3.33; 7000 5.22 / 4.93, 4.46 / 4.31; 10000 7.58 / 6.29, 6.51 / 5.39.
    if (G.nx <= 3 * 608) launch_stages<4>(s, G, cs);
    else launch_stages<16>(s, G, cs);
    return;
  }
  const unsigned gf = unsigned((G.nx + 1 + kThreads - 1) / kThreads);
  const unsigned gc = unsigned((G.nx + kThreads - 1) / kThreads);
  float* F = static_cast<float*>(s->work);
  k_begin_step<<<1, 1, 0, cs>>>(s->dstate);
  for (int stage = 1; stage <= 3; ++stage) {
    k1_flux_f<<<gf, kThreads, 0, cs>>>(G, s->q, F, s->dstate);
    k1_update_f<<<gc, kThreads, 0, cs>>>(G, stage, F, s->q, s->q0, s->dstate);
  }
  k_end_step<<<1, 1, 0, cs>>>(s->dstate);
}

// A 1D step is 3 or 8 small launches whose CPU launch cost exceeds their GPU time; runs of
// kGraphSteps steps are captured once into a graph (the solver's buffers are fixed) and replayed.
constexpr int kGraphSteps = 16;

void launch_steps(hteno_solver* s, const Geo1& G, int n, cudaStream_t cs) {
  for (int k = 0; k < n; ++k) launch_step(s, G, cs);
}

cudaError_t ensure_graph(hteno_solver* s, const Geo1& G) {
  if (s->step_graph) return cudaSuccess;
  cudaStream_t cap;
  cudaError_t e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  cudaGraph_t g = nullptr;
  e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    launch_steps(s, G, kGraphSteps, cap);
    e = cudaStreamEndCapture(cap, &g);
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&s->step_graph, g, 0);
  if (g) cudaGraphDestroy(g);
  cudaStreamDestroy(cap);
  return e;
}

}  // namespace

int fv1d_setup(hteno_solver* s) {
  if (upload_const(&g_mask, &g_mu, c_dev, g_dev) != cudaSuccess)
    return set_error(s, HTENO_ERR_CUDA, "constant upload failed");
  s->work_bytes = s->cfg.precision == HTENO_PREC_FP64 ? kWorkArrays * size_t(s->cfg.nx) * sizeof(double)
                                                       : 3 * size_t(s->cfg.nx + 1) * sizeof(float);
  cudaError_t e = cudaMalloc(&s->work, s->work_bytes);
  if (e != cudaSuccess) return cuda_error(s, e, "work buffer");
  s->launches_per_step = s->cfg.precision == HTENO_PREC_FP64 ? 3 : 2 + 3 * 2;
  return HTENO_OK;
}

int fv1d_prepare(hteno_solver* s) {
  const Geo1 G = geo1_of(s);
  double* prim = s->cfg.precision == HTENO_PREC_FP64 ? static_cast<double*>(s->work) + 3 * size_t(G.nx) : nullptr;
  k1_init<<<unsigned((G.nx + 127) / 128), 128, 0, s->stream>>>(G, s->q, prim, s->dstate);
  return cuda_error(s, cudaGetLastError(), "k1_init");
}

int fv1d_harvest(hteno_solver* s, double p, unsigned long long seed, uint16_t* X, uint8_t* Y,
                 long cap, unsigned long long* count) {
  const Geo1 G = geo1_of(s);
  k1_harvest<<<unsigned((G.nx + 1 + kThreads - 1) / kThreads), kThreads, 0, s->stream>>>(
      G, s->q, p, seed, X, Y, cap, count);
  return cuda_error(s, cudaGetLastError(), "harvest");
}

int fv1d_kxrcf(hteno_solver* s, uint8_t* flags) {
  const Geo1 G = geo1_of(s);
  const double crm = pow(G.dx / 2.0, 1.5);  // circleRadMod (FV_System1D.cpp:19)
  k1_kxrcf<<<unsigned((G.nx + kThreads - 1) / kThreads), kThreads, 0, s->stream>>>(G, s->q, crm, flags);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  return cuda_error(s, e, "kxrcf");
}

int fv1d_step_async(hteno_solver* s, int nsteps) {
  const Geo1 G = geo1_of(s);
  int left = nsteps;
  if (!s->timing && nsteps >= kGraphSteps) {  // per-kernel timing needs the plain launches
    const cudaError_t e = ensure_graph(s, G);
    if (e != cudaSuccess) return cuda_error(s, e, "fv1d step graph");
    for (; left >= kGraphSteps; left -= kGraphSteps) {
      const cudaError_t el = cudaGraphLaunch(s->step_graph, s->stream);
      if (el != cudaSuccess) return cuda_error(s, el, "fv1d graph launch");
    }
  }
  launch_steps(s, G, left, s->stream);
  return cuda_error(s, cudaGetLastError(), "fv1d step launch");
}

}  // namespace hteno
