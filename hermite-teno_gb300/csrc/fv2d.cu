// FV::System2D on the GPU (FV_System2D.cpp:363-651): characteristic TENO5 per direction,
// transverse three-point Gauss-Legendre WENO5-JS along each face, HLLC or characteristic
// Rusanov at the Gauss points, SSP-RK3.  Host dispatch of the two precisions:
//
//   plain FP64 (fv2d_fp64.cu): bit-reproducible; 5 launches per stage (faces x/y, flux x/y,
//     update) through per-face work arrays, or one fused launch per stage over 32 x 32 tiles
//     (hteno_set_fp64_fused, the same bits);
//   mixed (fv2d_fused.cu): reconstruction and fluxes in float, state and RK accumulation in
//     double; one fused launch per stage over tiles held in shared memory.
//
// One step = k_begin_step, 3 stages, k_end_step.  The host never synchronises inside
// hteno_step: dt, t and the stop flag live on the device.
#include "fv2d_common.cuh"

namespace hteno {
namespace {

#include "common_kernels.cuh"

}  // namespace

int fv2d_setup(hteno_solver* s) {
  if (fv2d_fp64_setup(s) != HTENO_OK) return HTENO_ERR_CUDA;
  const int nx = s->cfg.nx, ny = s->cfg.ny;
  if (s->cfg.precision == HTENO_PREC_MIXED) {
    const int rc = fv2d_fused_setup(s);
    if (rc != HTENO_OK) return rc;
    s->work_bytes = fv2d_fused_work_bytes(nx, ny);
    s->launches_per_step = 2 + 3;
  } else {
    s->work_bytes = work_bytes<double>(nx, ny);
    s->launches_per_step = 2 + 3 * (5 + (s->uniform_skip ? 1 : 0));  // + the uniform-region test
  }
  cudaError_t e = cudaMalloc(&s->work, s->work_bytes);
  if (e != cudaSuccess) return cuda_error(s, e, "work buffer");
  return HTENO_OK;
}

int fv2d_prepare(hteno_solver* s) {
  const Geo G = geo_of(s);
  if (s->cfg.precision == HTENO_PREC_MIXED)
    return fv2d_fused_prepare(s, G, static_cast<double*>(s->work));
  fv2d_fp64_prim(s, G, carve<double>(s->work, G.nx, G.ny), s->q, s->dstate, 1);
  return cuda_error(s, cudaGetLastError(), "primitives");
}

namespace {

void launch_step(hteno_solver* s, const Geo& G) {
  launch_early(s->early, k_begin_step, 1, 1, 0, s->stream, s->dstate);
  if (s->cfg.precision == HTENO_PREC_MIXED) {
    fv2d_fused_step(s, G, static_cast<double*>(s->work));
  } else {
    const Work<double> W = carve<double>(s->work, G.nx, G.ny);
    if (s->fused64) fv2d_fp64_fused_step(s, G, W);
    else for (int stage = 1; stage <= 3; ++stage) fv2d_fp64_stage(s, G, W, stage, s->q, nullptr);
  }
  launch_early(s->early, k_end_step, 1, 1, 0, s->stream, s->dstate);
}

// A plain FP64 step of a small grid is 20 launches on two streams of ~10-30 us each, which the host
// issues hardly faster than they run: runs of kGraphSteps steps are captured once into a graph (the
// solver's buffers are fixed; dt, t and the stop live on the device) and replayed.  Larger grids'
// launches outlast their issue.  64 x 48, 24 steps with state copies: 7.5 -> 6.2 ms with the blocks of
// update_threads.  Eight steps, launched / replayed, four quadrants and periodic waves: 64^2 2.70 / 2.43, 2.52 / 2.25
// ms; 128^2 6.40 / 6.15, 5.30 / 5.07; 181^2 10.76 / 10.69, 9.81 / 9.54; 200^2 12.48 / 12.42, 12.02 / 11.79;
// 230^2 16.35 / 16.59, 13.93 / 14.63; 320^2 24.18 / 23.59, 25.79 / 25.57.
constexpr int kGraphSteps = 4;
constexpr size_t kGraphCells = size_t(1) << 15;

// (a stream that the caller is capturing takes the launches themselves)
bool capturing(const hteno_solver* s) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(s->stream, &c) != cudaSuccess || c != cudaStreamCaptureStatusNone;
}
bool graphed(const hteno_solver* s) {
  return s->cfg.precision == HTENO_PREC_FP64 && !s->fused64 && !s->timing && s->ncell <= kGraphCells && !capturing(s);
}

// While it lives, this thread may make calls that a capture elsewhere (the caller's, on another stream or in
// another thread) would refuse and be invalidated by: creating a stream, instantiating a graph.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

cudaError_t ensure_graph(hteno_solver* s, const Geo& G) {
  if (s->step_graph) return cudaSuccess;
  const RelaxedCapture relaxed;
  cudaStream_t cap, own = s->stream;
  cudaError_t e = cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking);
  if (e != cudaSuccess) return e;
  cudaGraph_t g = nullptr;
  e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    s->stream = cap;  // the side stream joins the capture through its fork event
    for (int k = 0; k < kGraphSteps; ++k) launch_step(s, G);
    s->stream = own;
    e = cudaStreamEndCapture(cap, &g);
  }
  if (e == cudaSuccess) e = cudaGraphInstantiate(&s->step_graph, g, 0);
  if (g) cudaGraphDestroy(g);
  cudaStreamDestroy(cap);
  return e;
}

}  // namespace

int fv2d_step_async(hteno_solver* s, int nsteps) {
  const Geo G = geo_of(s);
  int left = nsteps;
  if (graphed(s) && left >= kGraphSteps) {
    const cudaError_t e = ensure_graph(s, G);
    if (e != cudaSuccess) return cuda_error(s, e, "fv2d step graph");
    for (; left >= kGraphSteps; left -= kGraphSteps) {
      const cudaError_t el = cudaGraphLaunch(s->step_graph, s->stream);
      if (el != cudaSuccess) return cuda_error(s, el, "fv2d graph launch");
    }
  }
  // a mixed step is 5 kernels in one stream, each of which starts while the one before it ends (24 steps
  // of 96 x 80 with the small tiles: 1.88 -> 1.18 ms)
  s->early = s->cfg.precision == HTENO_PREC_MIXED && !s->timing && !capturing(s);
  for (; left > 0; --left) launch_step(s, G);
  s->early = false;
  return cuda_error(s, cudaGetLastError(), "fv2d step launch");
}

int fv2d_residual(hteno_solver* s, const double* q, double* rhs) {
  const Geo G = geo_of(s);
  if (s->cfg.precision == HTENO_PREC_MIXED) {
    fv2d_fused_residual(s, G, q, rhs);
  } else {
    Work<double> W = carve<double>(s->work, G.nx, G.ny);
    fv2d_fp64_prim(s, G, W, q, nullptr, 0);
    fv2d_fp64_stage(s, G, W, 0, q, rhs);
  }
  return cuda_error(s, cudaGetLastError(), "fv2d residual launch");
}

int fv2d_harvest_entry(hteno_solver* s, double p, unsigned long long seed, uint16_t* X, uint8_t* Y,
                       long cap, unsigned long long* count) {
  const Geo G = geo_of(s);
  return fv2d_harvest(s, G, carve<double>(s->work, G.nx, G.ny), p, seed, X, Y, cap, count);
}

}  // namespace hteno
