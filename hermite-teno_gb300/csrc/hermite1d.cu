// FVHermite::System1D on the GPU (FVHermite_System1D.cpp:183-405): periodic boundaries, LMPE
// troubled-cell detection, conditional derivative limiter, htenoi on troubled cells and linear
// Hermite reconstruction elsewhere, Rusanov + dRusanov, SSP-RK3, dt = cfl dx^(5/3) / max speed.
//
// The LMPE scan (:239-257) is sequential along x (a cell flagged by its left neighbour is
// skipped) and its flags live on the ghost-padded index space [0, nx + 2k) and are never reset;
// the limiter (:259-273) runs once per rhs over the padded range when any flag is set, updating
// the moments in place (a Gauss-Seidel sweep that also limits the left ghost first).  Both are one
// block: the scan's outcome follows from the cells' tests by bit operations on words of 32 cells,
// and the sweep runs in segments side by side (see kh1_sensor).  A face's FP64 work is spread over 8
// lanes; updates are one thread per cell.  In double the bit-reproducible functions
// (parity_math.cuh) are used; compiled with --fmad=false.
#include <type_traits>

#include "hermite_limit.cuh"
#include "hteno_internal.h"

namespace hteno {
namespace {

__constant__ DevConst c_dev;
__device__ DevConst g_dev;  // the same in global memory (double: par::ldk)
unsigned long long g_mask = 0;
std::mutex g_mu;

#include "common_kernels.cuh"

constexpr int kGhost = 4;  // k of FVHermite::System1D (:24)
constexpr int kS = 1;      // s (:25)

struct GeoH1 {
  int nx, nxx;
  double dx, area, gamma, g1, g3;  // g3 = gamma - 3 as the reference computes it
};

template <typename T>
struct WorkH1 {
  double* vl;            // [3][nx] limited moments (the solver's v keeps the unlimited ones)
  unsigned* words;       // [3][(nxx + 31) / 32] the LMPE scan's candidate cells, then its hits
  unsigned char* flags;  // [nxx][3] LMPE flags (persist)
  T* Fu;                 // [3][nx+1]
  T* Fv;                 // [3][nx+1]
};

template <typename T>
size_t work_bytes_h1(int nx) {
  const int nxx = nx + 2 * kGhost;
  return 3 * size_t(nx) * 8 + 3 * size_t((nxx + 31) / 32) * 4 + 3 * size_t(nxx) + 2 * 3 * size_t(nx + 1) * sizeof(T) + 256 * 5;
}

template <typename T>
WorkH1<T> carve_h1(void* base, int nx) {
  const int nxx = nx + 2 * kGhost;
  char* p = static_cast<char*>(base);
  auto take = [&](size_t bytes) {
    char* r = p;
    p += (bytes + 255) & ~size_t(255);
    return r;
  };
  WorkH1<T> w;
  w.vl = reinterpret_cast<double*>(take(3 * size_t(nx) * 8));
  w.words = reinterpret_cast<unsigned*>(take(3 * size_t((nxx + 31) / 32) * 4));
  w.flags = reinterpret_cast<unsigned char*>(take(3 * size_t(nxx)));
  w.Fu = reinterpret_cast<T*>(take(3 * size_t(nx + 1) * sizeof(T)));
  w.Fv = reinterpret_cast<T*>(take(3 * size_t(nx + 1) * sizeof(T)));
  return w;
}

__device__ __forceinline__ int wrap(int i, int n) {  // padded index -> interior (periodic)
  int m = i - kGhost;
  m %= n;
  return m < 0 ? m + n : m;
}

__device__ __forceinline__ void prim1(double g1, const double* q, double* w, double& h, double& sr) {
  w[0] = q[0];
  w[1] = q[1] / q[0];
  w[2] = (q[2] - 0.5 * q[1] * w[1]) * g1;
  h = (q[2] + w[2]) / w[0];
  sr = sqrt(fabs(w[0]));
}

__global__ void kh1_init(GeoH1 G, const double* __restrict__ q, StepState* st) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double ms = 0.0;
  if (i < G.nx) {
    double qq[3] = {q[i], q[G.nx + i], q[2 * G.nx + i]}, w[3], h, sr;
    prim1(G.g1, qq, w, h, sr);
    ms = par::max_speed1(G.gamma, w[1], w[2], par::den_of(w[0]));
  }
  block_max_to(ms, &st->maxbits);
}

// Of the candidate cells of a word (bit k: cell k passes the LMPE test and carries no flag yet), those
// the scan from left to right hits: every other one of a run of candidates, from its first on (a hit
// flags its right neighbour, which the scan then skips).  hit: whether the cell before bit 0 was hit.
__device__ __forceinline__ unsigned lmpe_hits(unsigned c, bool hit) {
  if (hit) c &= ~1u;
  const unsigned even = (c & ~(c << 1)) & 0x55555555u;  // first bits of the runs that start at even bits
  const unsigned re = c & ~(c + even);                  // those runs (the carry clears each)
  return (re & 0x55555555u) | (c & ~re & 0xaaaaaaaau);
}

// The limiter's cell in the solver's precision: in double LimitSweep (hermite_limit.cuh), in float
// hermiteLimiter as it stands.
template <typename T>
struct LimitSweep1;
template <>
struct LimitSweep1<double> : LimitSweep<double> {
  using LimitSweep<double>::LimitSweep;
  __device__ __forceinline__ double cell(double dl, bool again) { return again && flat() ? at_flat(dl) : at(dl); }
};
template <>
struct LimitSweep1<float> {
  const HermiteK<float>& K;
  float u0, u1, u2, d2;
  __device__ __forceinline__ LimitSweep1(const HermiteK<float>& k, float ul, float uc) : K(k), u1(ul), u2(uc) {}
  __device__ __forceinline__ void next(float ur, float dr) {
    u0 = u1;
    u1 = u2;
    u2 = ur;
    d2 = dr;
  }
  __device__ __forceinline__ float cell(float dl, bool) const {
    const float u[3] = {u0, u1, u2}, d[3] = {dl, 0.f, d2};
    return hermite_limiter(K, u, d);
  }
};

// LMPE + conditional limiter, one block of 128 threads: one warp per SM sub-partition, as many as its
// FP64 unit (64 cycles a warp instruction) can use.  The limiter's sweep along the padded line is cut
// into kSeg segments per field that sweep side by side, each from a guess of its left neighbour's
// value, and again from the neighbour's result while that came out with other bits than were used: the
// bits of the one sweep (see kh_limit of the 2D scheme).  The limited moments go to W.vl, or the
// unlimited ones where no flag is set.  At 320 cells in double 1930 -> 157 us per launch: one thread
// per field walked the line before.
constexpr int kSensorThreads = 128, kSeg = kSensorThreads / 3, kWarm = 24;

template <typename T>
__global__ void __launch_bounds__(kSensorThreads) kh1_sensor(GeoH1 G, HermiteK<T> K, const double* __restrict__ q,
                                                             const double* __restrict__ v, WorkH1<T> W,
                                                             const StepState* st) {
  __shared__ T last[kSensorThreads];
  if (st->done) return;
  const int n = G.nx, nxx = G.nxx, nw = (nxx + 31) / 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  unsigned char* fl = W.flags;
  auto at = [&](int i) {  // padded index -> interior (periodic), |offset| <= kGhost
    const int m = i - kGhost;
    return m < 0 ? m + n : m >= n ? m - n : m;
  };
  // LMPE: each unflagged cell's test, a word of 32 cells per warp and turn
  bool any = false;
  for (int w = wid; w < 3 * nw; w += kSensorThreads / 32) {
    const int e = w / nw, i = (w - e * nw) * 32 + lane;
    bool cand = false;
    if (i >= kS + 1 && i < nxx - kS - 1) {
      if (fl[3 * i + e]) {
        any = true;
      } else {
        const double* u = q + size_t(e) * n;
        const double um = u[at(i - 1)], u0 = u[at(i)], up = u[at(i + 1)];
        const double A = fabs(-um + 2.0 * u0 - up) / 2.0;
        if (A > 0.5 * G.dx) {
          const double xc = (-2. * um + 3. * u0 - up) / (-um + 2.0 * u0 - up) * G.dx;
          cand = 0.0 <= xc && xc <= 3. * G.dx;
        }
      }
    }
    const unsigned word = __ballot_sync(0xffffffffu, cand);
    if (lane == 0) W.words[w] = word;
  }
  __syncthreads();
  if (tid < 3) {
    bool hit = false;
    for (int w = tid * nw; w < (tid + 1) * nw; ++w) {
      const unsigned h = lmpe_hits(W.words[w], hit);
      W.words[w] = h;
      any |= h != 0u;
      hit = h >> 31;
    }
  }
  any = __syncthreads_or(any);
  for (int w = wid; w < 3 * nw; w += kSensorThreads / 32) {
    const int e = w / nw, i = (w - e * nw) * 32 + lane;
    if (W.words[w] >> lane & 1u) {
      fl[3 * (i - 1) + e] = 1;
      fl[3 * i + e] = 1;
      fl[3 * (i + 1) + e] = 1;
    }
  }
  if (!any) {
    for (int k = tid; k < 3 * n; k += kSensorThreads) W.vl[k] = v[k];
    return;
  }
  // the sweep over the padded cells kGhost - 1 .. nx + kGhost - 1 (the left ghost, then the interior;
  // the reference also limits the first right ghost, which nothing reads)
  const int e = tid / kSeg, seg = tid - e * kSeg;
  const int first = kGhost - 1, cells = n + 1, len = (cells + kSeg - 1) / kSeg;
  const int c0 = first + min(cells, seg * len), c1 = min(first + cells, c0 + len);
  const bool live = e < 3 && c0 < c1;
  const double *u = q + size_t(e) * n, *d = v + size_t(e) * n;
  double* out = W.vl + size_t(e) * n;
  T used = T(0);
  auto sweep = [&](T dl, bool again) {
    LimitSweep1<T> s(K, T(u[at(c0 - 1)]), T(u[at(c0)]));
    for (int i = c0; i < c1; ++i) {
      s.next(T(u[at(i + 1)]), T(d[at(i + 1)]));
      dl = s.cell(dl, again);
      if (i < kGhost) continue;  // the ghost (never swept again: its left neighbour is given)
      if (again && same_bits(double(dl), out[i - kGhost])) return;
      out[i - kGhost] = double(dl);
    }
    last[tid] = dl;
  };
  if (live) {
    used = T(d[at(c0 - 1)]);
    if constexpr (std::is_same<T, double>::value) {
      if (c0 - kWarm > first) {  // the guess: the float sweep of the cells before
        LimitSweep<float> s(K, float(u[at(c0 - kWarm - 1)]), float(u[at(c0 - kWarm)]));
        float x = float(d[at(c0 - kWarm - 1)]);
        for (int i = c0 - kWarm; i < c0; ++i) {
          s.next(float(u[at(i + 1)]), float(d[at(i + 1)]));
          x = s.at(x);
        }
        if (fabsf(x) <= 3.4e38f) used = double(x);
      }
    }
    sweep(used, false);
  }
  for (int pass = 1; pass < kSeg; ++pass) {
    __syncthreads();
    const T left = live && seg ? last[tid - 1] : used;
    const bool redo = live && !same_bits(left, used);
    if (!__syncthreads_or(redo)) break;
    if (redo) {
      used = left;
      sweep(left, true);
    }
  }
}

// face f in [0, nx] between interior cells f-1 and f (padded cell f + k - 1 and its neighbour),
// mixed precision
__global__ void kh1_faces_f(GeoH1 G, HermiteK<float> K, const double* __restrict__ q, WorkH1<float> W,
                            const StepState* st) {
  if (st->done) return;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = G.nx;
  if (f > n) return;
  const int ip = f + kGhost - 1;  // padded index of the left cell
  const double* v = W.vl;
  double qa[3], qb[3], wa[3], wb[3], ha, hb, sa, sb;
  const int ca = wrap(ip, n), cb = wrap(ip + 1, n);
  for (int c = 0; c < 3; ++c) {
    qa[c] = q[c * n + ca];
    qb[c] = q[c * n + cb];
  }
  prim1(G.g1, qa, wa, ha, sa);
  prim1(G.g1, qb, wb, hb, sb);
  float fu[3], fv[3];
  const Roe1<float> R = roe1<float>(float(G.g1), float(sa), float(wa[1]), float(ha), float(sb), float(wb[1]), float(hb));
  float A[3][4], B[3][4];
  for (int m = 0; m < 4; ++m) {
    const int c = wrap(ip - 1 + m, n);
    float a3[3] = {float(q[c]), float(q[n + c]), float(q[2 * n + c])};
    float b3[3] = {float(v[c]), float(v[n + c]), float(v[2 * n + c])};
    float ca3[3], cb3[3];
    roe1_left(R, a3, ca3);
    roe1_left(R, b3, cb3);
    for (int r = 0; r < 3; ++r) {
      A[r][m] = ca3[r];
      B[r][m] = cb3[r];
    }
  }
  float cl[4][3];
  for (int r = 0; r < 3; ++r) {
    float o[4];
    hermite_recon(c_dev, K, W.flags[3 * ip + r] ? 1 : 2, A[r], B[r], o);
    for (int a = 0; a < 4; ++a) cl[a][r] = o[a];
  }
  float X[4][3];
  for (int a = 0; a < 4; ++a) roe1_right(R, cl[a], X[a]);
  rusanov1(float(G.gamma), float(G.g1), R, X[0], X[1], fu);
  drusanov1(float(G.gamma), float(G.g1), R, X[0], X[1], X[2], X[3], fv);
  for (int c = 0; c < 3; ++c) {
    W.Fu[c * (n + 1) + f] = fu[c];
    W.Fv[c * (n + 1) + f] = fv[c];
  }
}

// The FP64 faces: 8 lanes per face, lane r + 4 s (r < 3) projects characteristic field r and
// reconstructs side s's value and derivative; lane 0 gathers the twelve values and computes the
// fluxes.  A line has a few hundred faces: the FP64 units take 64 cycles per warp instruction however
// many lanes are active, so a face's instructions in sequence set the time, and its lanes' warps
// spread over more of the chip.
__global__ void __launch_bounds__(64) kh1_faces(GeoH1 G, HermiteK<double> K, const double* __restrict__ q,
                                                WorkH1<double> W, const StepState* st) {
  if (st->done) return;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = G.nx, l = gid & 7, r = l & 3, side = l >> 2;
  const bool live = (gid >> 3) <= n;
  const int f = live ? gid >> 3 : n;  // lanes past the last face compute that face, store nothing
  const int ip = f + kGhost - 1;      // padded index of the left cell
  double qa[3], qb[3], wa[3], wb[3], ha, hb, sa, sb;
  const int ca = wrap(ip, n), cb = wrap(ip + 1, n);
  for (int c = 0; c < 3; ++c) {
    qa[c] = q[c * n + ca];
    qb[c] = q[c * n + cb];
  }
  prim1(G.g1, qa, wa, ha, sa);
  prim1(G.g1, qb, wb, hb, sb);
  par::fp R[9], L[9];
  par::eig1(G.g1, sa, wa[1], ha, sb, wb[1], hb, R, L);
  double val = 0.0, der = 0.0;
  if (r < 3) {
    const par::fp l0 = r == 0 ? L[0] : r == 1 ? L[3] : L[6];
    const par::fp l1 = r == 0 ? L[1] : r == 1 ? L[4] : L[7];
    const par::fp l2 = r == 0 ? L[2] : r == 1 ? L[5] : L[8];
    par::fp A[3], B[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const int c = wrap(ip - 1 + side + m, n);
      const par::fp a3[3] = {q[c], q[n + c], q[2 * n + c]};
      const par::fp b3[3] = {W.vl[c], W.vl[n + c], W.vl[2 * n + c]};
      A[m] = par::dot3(l0, l1, l2, a3);  // row r of par::mv3
      B[m] = par::dot3(l0, l1, l2, b3);
    }
    par::hermite_side(g_dev, K, W.flags[3 * ip + r] ? 1 : 2, A, B, side, val, der);
  }
  const int base = int(threadIdx.x & 31u) & ~7;
  par::fp cl[4][3];  // u-, u+, d-, d+
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    cl[0][k] = __shfl_sync(0xffffffffu, val, base + k);
    cl[1][k] = __shfl_sync(0xffffffffu, val, base + 4 + k);
    cl[2][k] = __shfl_sync(0xffffffffu, der, base + k);
    cl[3][k] = __shfl_sync(0xffffffffu, der, base + 4 + k);
  }
  if (l != 0 || !live) return;
  par::fp X[4][3], fu[3], fv[3];
  for (int a = 0; a < 4; ++a) par::mv3(R, cl[a], X[a]);
  const par::Sides1 S = par::sides1_of(G.gamma, G.g1, X[0], X[1]);
  par::rusanov1(S, L, R, X[0], X[1], fu);
  par::drusanov1(G.gamma, G.g1, G.g3, S, L, R, X[0], X[1], X[2], X[3], fv);
  for (int c = 0; c < 3; ++c) {
    W.Fu[c * (n + 1) + f] = fu[c].v;
    W.Fv[c * (n + 1) + f] = fv[c].v;
  }
}

template <typename T>
__global__ void kh1_update(GeoH1 G, int stage, WorkH1<T> W, double* __restrict__ q,
                           double* __restrict__ q0, double* __restrict__ v,
                           double* __restrict__ v0, StepState* st) {
  if (st->done) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int n = G.nx;
  double ms = 0.0;
  int bad = 0;
  if (i < n) {
    const double dt = st->dt;
    double qn[3];
    for (int c = 0; c < 3; ++c) {
      const double ru = (double(W.Fu[c * (n + 1) + i]) - double(W.Fu[c * (n + 1) + i + 1])) / G.area;
      const double rv = (double(W.Fv[c * (n + 1) + i]) - double(W.Fv[c * (n + 1) + i + 1])) / G.area;
      const size_t o = size_t(c) * n + i;
      double bq, bv, cq = q[o], cv;
      if (stage == 1) {
        bq = cq; bv = W.vl[o];  // save() after the first rhs: limited moments
        q0[o] = bq; v0[o] = bv;
        cv = bv;
      } else {
        bq = q0[o]; bv = v0[o];
        cv = v[o];  // the unlimited stage value
      }
      qn[c] = par::rk3(bq, cq, ru, dt, stage);
      const double nv = par::rk3(bv, cv, rv, dt, stage);
      q[o] = qn[c];
      v[o] = nv;
    }
    double w[3], h, sr;
    prim1(G.g1, qn, w, h, sr);
    if (stage == 3) ms = par::max_speed1(G.gamma, w[1], w[2], par::den_of(w[0]));
    bad = (isnan(qn[0]) || isnan(qn[1]) || isnan(qn[2])) ? 1 : 0;
    bad |= (qn[0] <= 0.0 || w[2] <= 0.0) ? 2 : 0;
  }
  if (stage == 3) block_max_to(ms, &st->maxbits);
  if (bad) atomicOr(&st->status, bad);
}

GeoH1 geo_of(const hteno_solver* s) {
  GeoH1 G;
  G.nx = s->cfg.nx;
  G.nxx = s->cfg.nx + 2 * kGhost;
  G.dx = s->dx;
  G.area = s->dx;
  G.gamma = s->cfg.gamma;
  G.g1 = s->cfg.gamma - 1.0;
  G.g3 = s->cfg.gamma - 3.0;
  return G;
}

template <typename T>
void launch_step(hteno_solver* s, const GeoH1& G) {
  cudaStream_t cs = s->stream;
  const WorkH1<T> W = carve_h1<T>(s->work, G.nx);
  const HermiteK<T> K = make_hermite_k<T>(s->dx);
  const unsigned gc = unsigned((G.nx + 63) / 64);
  k_begin_step<<<1, 1, 0, cs>>>(s->dstate);
  for (int stage = 1; stage <= 3; ++stage) {
    kh1_sensor<T><<<1, kSensorThreads, 0, cs>>>(G, K, s->q, s->v, W, s->dstate);
    if constexpr (std::is_same<T, double>::value)
      kh1_faces<<<unsigned((8 * (G.nx + 1) + 63) / 64), 64, 0, cs>>>(G, K, s->q, W, s->dstate);
    else
      kh1_faces_f<<<unsigned((G.nx + 1 + 63) / 64), 64, 0, cs>>>(G, K, s->q, W, s->dstate);
    kh1_update<T><<<gc, 64, 0, cs>>>(G, stage, W, s->q, s->q0, s->v, s->v0, s->dstate);
  }
  k_end_step<<<1, 1, 0, cs>>>(s->dstate);
}

}  // namespace

int hermite1d_setup(hteno_solver* s) {
  if (upload_const(&g_mask, &g_mu, c_dev, g_dev) != cudaSuccess)
    return set_error(s, HTENO_ERR_CUDA, "constant upload failed");
  s->work_bytes = s->cfg.precision == HTENO_PREC_MIXED ? work_bytes_h1<float>(s->cfg.nx)
                                                       : work_bytes_h1<double>(s->cfg.nx);
  cudaError_t e = cudaMalloc(&s->work, s->work_bytes);
  if (e != cudaSuccess) return cuda_error(s, e, "work buffer");
  cudaMemset(s->v, 0, s->ncell * 3 * sizeof(double));
  s->launches_per_step = 2 + 3 * 3;
  return HTENO_OK;
}

int hermite1d_prepare(hteno_solver* s) {
  const GeoH1 G = geo_of(s);
  // a new initial state starts with cleared troubled-cell flags (fresh storage in the reference)
  unsigned char* flags = s->cfg.precision == HTENO_PREC_MIXED ? carve_h1<float>(s->work, G.nx).flags
                                                              : carve_h1<double>(s->work, G.nx).flags;
  cudaMemsetAsync(flags, 0, 3 * size_t(G.nxx), s->stream);
  kh1_init<<<unsigned((G.nx + 127) / 128), 128, 0, s->stream>>>(G, s->q, s->dstate);
  return cuda_error(s, cudaGetLastError(), "kh1_init");
}

int hermite1d_step_async(hteno_solver* s, int nsteps) {
  const GeoH1 G = geo_of(s);
  for (int n = 0; n < nsteps; ++n) {
    if (s->cfg.precision == HTENO_PREC_MIXED) launch_step<float>(s, G);
    else launch_step<double>(s, G);
  }
  return cuda_error(s, cudaGetLastError(), "hermite1d step launch");
}

}  // namespace hteno
