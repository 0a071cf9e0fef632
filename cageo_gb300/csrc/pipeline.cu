// pipeline.cu -- the Monte Carlo loop of src/main.cpp:180-283 as one object
// that owns its device buffers.
//
// A realization is: noise (Philox) -> fused convolution + realistic DEM +
// burning + quantization (front) -> pit fill -> routing -> tracing ->
// border counts.  In exact mode the front does not quantize and the fill,
// routing and tracing follow the reference's GPU path instead of its CPU
// path.  The launch sequence of a step -- one realization, or several stacked
// one above the other -- reads the realization number from device memory, so it
// is captured once in a CUDA graph and replayed; the data-dependent loops (fill
// passes, flat BFS layers, pointer jumps) run inside persistent kernels and
// need no host round trip.  Counts accumulate in uint32.
//
// The fused front uses a burn code precomputed from the stream raster.  It
// flags a realization where that code may differ from the reference's
// in-place burning (a stream cell whose realistic elevation equals NODATA);
// such a realization is not counted by the fast path and is recomputed with
// the stage kernels, which follow the reference step by step.  With a
// NODATA of 0 every realization takes the stage path.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>
#include <unistd.h>
#include "common.cuh"
#include "guard.h"
#include "front.cuh"
#include "pitfill.cuh"
#include "routing.cuh"

namespace cageo {
cageo_status launch_noise(float* d, int64_t n, uint64_t seed, uint32_t realization,
                          const uint32_t* dreal, float mean, float sd, cudaStream_t s, int slabs);
cageo_status launch_front(const float* noise, int W, int H, int model, const float* filt,
                          int r, const FrontParams& fp, cudaStream_t s, int tile, int slabs);
bool conv_tile_applies(int model, int r, int tile);
cageo_status launch_burn_code(const float* streams, uint8_t* code, int W, int H,
                              float nodata_stream, int bevel, float* factor_out,
                              cudaStream_t s);
cageo_status launch_realistic(const float* dem, float* field, int64_t n, float nodata,
                              cudaStream_t s);
cageo_status launch_burn_stage(const float* src, float* dst, const float* streams, int W,
                               int H, int bevel, float nodata_dem, float nodata_stream,
                               cudaStream_t s);
cageo_status launch_to_bytes(const float* in, uint8_t* out, int64_t n, unsigned int* mm,
                             cudaStream_t s);
cageo_status ws_infer(const float* params, const float* v, float* warm, float* depth, int W,
                      int H, float nodata, float threshold, cudaStream_t s);

// Layout of the device scalars (cageo_pipeline::dscal).
constexpr int kMaxStack = 64;               // realizations of a step
constexpr int kErrors = 1;                  // the run's first errors (keep_errors)
constexpr int kFlags = 4;                   // the step's anomaly flags
constexpr int kRedo = kFlags + kMaxStack;   // realizations to redo
constexpr unsigned int kMaxRedo = 4096;

// The error words of a step's fill, routing and tracing, and the word that says
// whether the fill needs the wide resolution.
struct StepErrors {
  const unsigned int *fill, *route, *trace, *wide;
};
constexpr uint32_t kWideSeen = 1u << 24;  // in dscal[kErrors]

// One thread at the end of a step: the next step's start clears the stages'
// error words, so the first step of a run that left any is kept, a byte per
// stage, until the host reads it at the run's end, and kWideSeen beside it.
__device__ __forceinline__ void keep_errors(const StepErrors& e, uint32_t* kept) {
  const uint32_t now = min(*e.fill, 255u) | min(*e.route, 255u) << 8 | min(*e.trace, 255u) << 16;
  const bool wide = *e.wide != 0u;
  if (!now && !wide) return;
  const uint32_t was = *kept;
  *kept = (was & (kWideSeen - 1u) ? was : was | now) | (wide ? kWideSeen : 0u);
}

__global__ void keep_errors_kernel(StepErrors e, uint32_t* kept) { keep_errors(e, kept); }

// End of a step of `count` realizations: list the flagged ones (they were not
// counted), clear their flags, keep the stages' errors and advance the device
// realization counter.
__global__ void realization_end_kernel(uint32_t* real, int* anomaly, uint32_t* redo,
                                       unsigned int* nredo, unsigned int count, StepErrors errors,
                                       uint32_t* kept) {
  for (unsigned int j = threadIdx.x; j < count; j += blockDim.x) {
    if (anomaly[j]) {
      const unsigned int k = atomicAdd(nredo, 1u);
      if (k < kMaxRedo) redo[k] = *real + j;
      anomaly[j] = 0;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    keep_errors(errors, kept);
    *real += count;
  }
}

// Order-independent 64-bit digest of a float grid: the wrapping sum over
// cells of a SplitMix64 finalizer of (cell index, value bits).  The
// checkpoint records it so that a resume onto other input grids is refused.
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void grid_digest_kernel(const float* __restrict__ g, int64_t n,
                                   unsigned long long salt, unsigned long long* out) {
  unsigned long long h = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    h += mix64(((unsigned long long)i * 0x9E3779B97F4A7C15ull) ^
               ((unsigned long long)__float_as_uint(g[i]) << 32) ^ salt);
  for (int o = 16; o; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, h);
}

// Bound by the copy (8 bytes a cell): 16 bytes a thread where `out` is aligned.
__global__ void __launch_bounds__(256) counts_to_float_kernel(const uint32_t* __restrict__ c,
                                                              float* __restrict__ f, int64_t n,
                                                              int aligned) {
  const int64_t base = (int64_t)blockIdx.x * 2048 + threadIdx.x * 4;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int64_t i = base + k * 1024;
    if (aligned && i + 4 <= n) {
      const uint4 v = *reinterpret_cast<const uint4*>(c + i);
      *reinterpret_cast<float4*>(f + i) = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
    } else {
      for (int64_t j = i; j < i + 4 && j < n; j++) f[j] = (float)c[j];
    }
  }
}

cageo_status counts_to_float(const uint32_t* c, float* f, int64_t n, cudaStream_t s) {
  counts_to_float_kernel<<<(unsigned)((n + 2047) / 2048), 256, 0, s>>>(c, f, n,
                                                                     ((uintptr_t)f & 15u) == 0);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

}  // namespace cageo

using namespace cageo;

struct cageo_pipeline {
  cageo_pipeline_config cfg{};
  int W = 0, H = 0;
  int64_t N = 0;
  int radius = 0;
  cudaStream_t stream = nullptr;
  float *dem = nullptr, *streams = nullptr, *noise = nullptr, *q = nullptr, *filled = nullptr,
        *filter = nullptr, *tmp = nullptr;
  uint8_t* code = nullptr;
  int8_t* dir = nullptr;
  int* label = nullptr;
  uint32_t* counts = nullptr;
  void *fill_ws = nullptr, *route_ws = nullptr, *trace_ws = nullptr;
  FillWork fw;
  RouteWork rw;
  TraceWork tw;
  // device scalars: [0] realization counter, [1] the run's first errors, [2]
  // nredo, [3] the run's last realization (the one whose labels are kept),
  // [4..] the anomaly flags of a step's slabs, then the redo list
  uint32_t* dscal = nullptr;
  FrontParams fp{};
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  bool graph_ok = false;
  int64_t stats[25] = {};
  // Learned warm start (exact mode only): parameters, warm surface, and the
  // fill's warm-start counters accumulated on the device (9 entries, see
  // fill_accumulate_warm_stats).
  float* ws_params = nullptr;
  float* warm = nullptr;
  unsigned long long* ws_acc = nullptr;
  float ws_threshold = 0.0f;
  // Digest of the DEM and stream grids (grid_digest_kernel), for checkpoints.
  unsigned long long input_digest = 0;
  // Stacked steps: `stack` realizations (the capacity; `step` of the last
  // step) one above the other through every stage -- q grids, filled grids,
  // directions, workspaces for W x K*H, each slab's minimum of q, and for
  // small grids their noise.  batch > 1: what cageo_pipeline_set_batch asked
  // for; 1: steps are sized by the grid (stack_of).
  int batch = 1;
  bool plain = false;  // batch 1 was asked for: one realization at a time
  int stack = 0, step = 0;
  int conv_tile = 0;  // the fused front's convolution tile shape (kConvTiles)
  float *qb = nullptr, *filledb = nullptr, *noiseb = nullptr;
  void *fill_ws_b = nullptr, *route_ws_b = nullptr, *trace_ws_b = nullptr;
  unsigned int* slab_min = nullptr;
  FillWork fwb;
  int8_t* dirb = nullptr;
  RouteWork rwb;
  TraceWork twb;
  int graph_k = 0;  // realizations of the captured step
  int last_k = 0;   // realizations of the last run's steps
  cudaGraph_t graph_b = nullptr;
  cudaGraphExec_t exec_b = nullptr;
  bool last_batched = false;  // the last realization ran in a stacked step (its top slab)
};

namespace {

void drop_step_graph(cageo_pipeline* p) {
  if (p->exec_b) cudaGraphExecDestroy(p->exec_b);
  if (p->graph_b) cudaGraphDestroy(p->graph_b);
  p->exec_b = nullptr;
  p->graph_b = nullptr;
  p->graph_k = 0;
}

void drop_graph(cageo_pipeline* p) {
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  p->exec = nullptr;
  p->graph = nullptr;
  p->graph_ok = false;
  drop_step_graph(p);
}

void free_stack(cageo_pipeline* p) {
  drop_step_graph(p);
  void* bufs[] = {p->qb, p->filledb, p->noiseb, p->fill_ws_b, p->slab_min, p->dirb,
                  p->route_ws_b, p->trace_ws_b};
  for (void* b : bufs)
    if (b) cudaFree(b);
  p->qb = p->filledb = p->noiseb = nullptr;
  p->fill_ws_b = p->route_ws_b = p->trace_ws_b = nullptr;
  p->slab_min = nullptr;
  p->dirb = nullptr;
  p->stack = p->step = 0;
  p->last_batched = false;
}

void free_all(cageo_pipeline* p) {
  free_stack(p);
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  void* bufs[] = {p->dem, p->streams, p->noise, p->q, p->filled, p->filter, p->tmp, p->code,
                  p->dir, p->label, p->counts, p->fill_ws, p->route_ws,
                  p->trace_ws, p->dscal, p->ws_params, p->warm, p->ws_acc};
  for (void* b : bufs)
    if (b) cudaFree(b);
  if (p->stream) cudaStreamDestroy(p->stream);
}

bool exact_mode(const cageo_pipeline* p) { return p->cfg.fill_mode == CAGEO_FILL_EXACT; }

// Fill, routing and tracing of the current realization in the pipeline's
// mode; p->q holds the (quantized or raw) burned realistic DEM.
// With the learned warm start (exact mode), the network's warm surface is
// inferred from q first; the fill verifies and repairs it itself.
cageo_status enqueue_fill(cageo_pipeline* p) {
  if (!exact_mode(p)) return fill_run(p->q, p->filled, p->fw, p->cfg.nodata_dem, p->stream);
  if (!p->ws_params)
    return fill_run_exact(p->q, p->filled, p->fw, p->cfg.nodata_dem, nullptr, p->stream);
  cageo_status st = ws_infer(p->ws_params, p->q, p->warm, nullptr, p->W, p->H, p->cfg.nodata_dem,
                             p->ws_threshold, p->stream);
  if (st) return st;
  if ((st = fill_run_exact(p->q, p->filled, p->fw, p->cfg.nodata_dem, p->warm, p->stream)))
    return st;
  return fill_accumulate_warm_stats(p->fw, p->ws_acc, p->stream);
}

cageo_status enqueue_route(cageo_pipeline* p) {
  return route_run(p->filled, p->dir, nullptr, p->rw, p->stream,
                   exact_mode(p) ? CAGEO_ROUTE_GPU_ORDER : CAGEO_ROUTE_CPU_COMPAT,
                   p->cfg.nodata_dem);
}

int trace_mode(const cageo_pipeline* p) {
  return exact_mode(p) ? CAGEO_TRACE_DEAD_END_ERROR : CAGEO_TRACE_CPU_COMPAT;
}

// Tracing whose labels are decoded by the border pass (one pass fewer);
// gate: skip the accumulation when set (null: always accumulate); every:
// write the labels whichever realization it is.
cageo_status enqueue_trace_border(cageo_pipeline* p, const int* gate, bool every) {
  cageo_status st = trace_run(p->dir, p->streams, p->code, p->label, p->tw, p->stream,
                              trace_mode(p), false);
  if (st) return st;
  return border_u32_from_state(p->tw, p->label, p->counts, gate, trace_mode(p), p->dscal,
                               every ? nullptr : p->dscal + 3, p->stream);
}

StepErrors step_errors(const FillWork& f, const RouteWork& r, const TraceWork& t) {
  return StepErrors{fill_error_word(f), route_error_word(r), trace_error_word(t),
                    fill_wide_word(f)};
}

// End of a step of `count` realizations in the given workspaces.
cageo_status enqueue_end(cageo_pipeline* p, const StepErrors& e, int count) {
  realization_end_kernel<<<1, 32, 0, p->stream>>>(p->dscal, (int*)p->dscal + kFlags,
                                                  p->dscal + kRedo, p->dscal + 2,
                                                  (unsigned int)count, e, p->dscal + kErrors);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

// What keep_errors kept of a run.
cageo_status kept_status(uint32_t kept) {
  if (!(kept & (kWideSeen - 1u))) return CAGEO_OK;
  const uint32_t fill = kept & 255u;
  if (fill) set_error("pit filling: %s", fill_error_text(fill));
  else if (kept >> 8 & 255u) set_error("flow routing: %s", route_error_text());
  else set_error("flow tracing: %s", trace_error_text());
  return CAGEO_ERR_NO_CONVERGENCE;
}

// Launch sequence of one realization on the fast path.  The realization
// number is read from dscal[0] by the noise kernel.
cageo_status enqueue_fast(cageo_pipeline* p) {
  cudaStream_t s = p->stream;
  const cageo_pipeline_config& c = p->cfg;
  cageo_status st;
  if ((st = fill_begin(p->fw, s))) return st;
  if ((st = launch_noise(p->noise, p->N, c.seed, 0, p->dscal, c.error_mean, c.error_stddev, s, 1)))
    return st;
  if ((st = launch_front(p->noise, p->W, p->H, c.filter_model, p->filter, p->radius, p->fp, s,
                         p->conv_tile, 1)))
    return st;
  if ((st = enqueue_fill(p))) return st;
  if ((st = enqueue_route(p))) return st;
  if ((st = enqueue_trace_border(p, (const int*)p->dscal + kFlags, false))) return st;
  return enqueue_end(p, step_errors(p->fw, p->rw, p->tw), 1);
}

// Launch sequence of one stacked step: p->step realizations from the device
// counter on, one above the other (slabs cannot exchange values: every slab's
// border cells are outlets of the fill and drain outward).  Every stage runs
// once over the stack; for grids above kStackNoise cells noise and front run
// slab by slab, which spares a noise grid per slab and loses nothing there (four
// at 4096^2: 4.00 ms slab by slab, 3.93 stacked).  The results equal single
// realizations bit for bit.
constexpr int64_t kStackNoise = (int64_t)1 << 24;

cageo_status enqueue_step(cageo_pipeline* p) {
  cudaStream_t s = p->stream;
  const cageo_pipeline_config& c = p->cfg;
  const int K = p->step;
  cageo_status st;
  if ((st = fill_begin(p->fwb, s))) return st;
  CAGEO_CUDA(cudaMemsetAsync(p->slab_min, 0xff, sizeof(unsigned int) * K, s));
  FrontParams fp = p->fp;
  fp.tseed = p->fwb.tseed;
  fp.tiles_x = p->fwb.tiles_x;
  const int each = p->noiseb ? K : 1;  // slabs per launch of noise and front
  for (int k = 0; k < K; k += each) {
    float* noise = p->noiseb ? p->noiseb : p->noise;
    if ((st = launch_noise(noise, p->N, c.seed, (uint32_t)k, p->dscal, c.error_mean,
                           c.error_stddev, s, each)))
      return st;
    fp.q = p->qb + (size_t)k * p->N;
    fp.min_ord = p->slab_min + k;
    fp.anomaly = p->fp.anomaly + k;
    fp.row0 = k * p->H;
    if ((st = launch_front(noise, p->W, p->H, c.filter_model, p->filter, p->radius, fp, s,
                           p->conv_tile, each)))
      return st;
  }
  if (exact_mode(p)) st = fill_run_exact(p->qb, p->filledb, p->fwb, c.nodata_dem, nullptr, s);
  else st = fill_run(p->qb, p->filledb, p->fwb, c.nodata_dem, s);
  if (st) return st;
  if ((st = route_run(p->filledb, p->dirb, nullptr, p->rwb, s,
                      exact_mode(p) ? CAGEO_ROUTE_GPU_ORDER : CAGEO_ROUTE_CPU_COMPAT,
                      c.nodata_dem)))
    return st;
  if ((st = trace_run(p->dirb, p->streams, p->code, p->label, p->twb, s, trace_mode(p), false)))
    return st;
  if ((st = border_u32_from_state(p->twb, p->label, p->counts, (const int*)p->dscal + kFlags,
                                  trace_mode(p), p->dscal, p->dscal + 3, s)))
    return st;
  return enqueue_end(p, step_errors(p->fwb, p->rwb, p->twb), K);
}

// The wide resolution is part of every fill as long as this lives.
struct WithWide {
  FillWork& w;
  const bool was;
  explicit WithWide(FillWork& fill) : w(fill), was(fill.wide) { w.wide = true; }
  ~WithWide() { w.wide = was; }
};

// Reference-order stage sequence for one realization (exact burning).
cageo_status run_stage_path(cageo_pipeline* p, uint32_t r) {
  cudaStream_t s = p->stream;
  const cageo_pipeline_config& c = p->cfg;
  cageo_status st;
  if ((st = fill_begin(p->fw, s))) return st;
  if ((st = launch_noise(p->noise, p->N, c.seed, r, nullptr, c.error_mean, c.error_stddev, s, 1)))
    return st;
  if ((st = cageo_convolve(p->noise, p->tmp, p->W, p->H, c.filter_model, p->filter, p->radius, s)))
    return st;
  if ((st = launch_realistic(p->dem, p->tmp, p->N, c.nodata_dem, s))) return st;
  if ((st = launch_burn_stage(p->tmp, p->q, p->streams, p->W, p->H, c.bevel_radius, c.nodata_dem,
                              c.nodata_stream, s)))
    return st;
  if (!exact_mode(p) && (st = fill_quantize_min(p->q, p->fw, c.nodata_dem, s))) return st;
  // In exact mode no stage kernel has set the fill's seeds.
  p->fw.seeded = !exact_mode(p);
  const WithWide wide(p->fw);
  st = enqueue_fill(p);
  p->fw.seeded = true;
  if (st) return st;
  if ((st = enqueue_route(p))) return st;
  if ((st = enqueue_trace_border(p, nullptr, true))) return st;
  keep_errors_kernel<<<1, 1, 0, s>>>(step_errors(p->fw, p->rw, p->tw), p->dscal + kErrors);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

// Largest filter radius a pipeline accepts (per-call filters included).
constexpr int kMaxRunRadius = 64;

template <typename T>
cageo_status dalloc(T** ptr, size_t bytes) {
  if (cudaMalloc((void**)ptr, bytes ? bytes : 16) == cudaSuccess) return CAGEO_OK;
  cudaGetLastError();
  scratch_trim();
  CAGEO_CUDA(cudaMalloc((void**)ptr, bytes ? bytes : 16));
  return CAGEO_OK;
}

cageo_status create_common(cageo_pipeline** out, const cageo_pipeline_config* cfg,
                           const float* dem, const float* streams, cudaMemcpyKind kind) {
  CAGEO_CHECK_ARG(out && cfg && dem && streams, "null argument");
  const int W = cfg->width, H = cfg->height;
  CAGEO_CHECK_ARG(valid_dims(W, H) && W >= 2 && H >= 2, "grid size");
  CAGEO_CHECK_ARG(W <= 65535 && H <= 65535, "width and height must be <= 65535");
  CAGEO_CHECK_ARG(cfg->filter_model == CAGEO_FILTER_GAUSSIAN ||
                      cfg->filter_model == CAGEO_FILTER_EXPONENTIAL,
                  "filter model");
  CAGEO_CHECK_ARG(cfg->bevel_radius >= 1 && cfg->bevel_radius <= 5, "bevel radius must be 1..5");
  CAGEO_CHECK_ARG(cfg->fill_mode == CAGEO_FILL_CPU_COMPAT || cfg->fill_mode == CAGEO_FILL_EXACT,
                  "fill mode");
  CAGEO_CHECK_ARG(cfg->cell_size > 0 && cfg->practical_range > 0, "range and cell size");
  const int r = cageo_filter_radius(cfg->practical_range, cfg->cell_size);
  CAGEO_CHECK_ARG(r >= 0 && r < W && r < H, "filter radius must be below the grid size");
  CAGEO_CHECK_ARG(r <= kMaxRunRadius, "filter radius above 64");
  const int L = 2 * r + 1;
  const int taps = cfg->filter_model == CAGEO_FILTER_GAUSSIAN ? L : L * L;
  std::vector<float> hf(taps);
  cageo_status st = cageo_filter_build(cfg->filter_model, cfg->practical_range, cfg->cell_size,
                                       r, hf.data());
  if (st) return st;
  auto* p = new (std::nothrow) cageo_pipeline();
  if (!p) {
    set_error("out of host memory for the pipeline object");
    return CAGEO_ERR_HOST;
  }
  p->cfg = *cfg;
  p->W = W;
  p->H = H;
  p->N = (int64_t)W * H;
  p->radius = r;
  auto fail = [&](cageo_status s) {
    free_all(p);
    delete p;
    return s;
  };
  if (cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking) != cudaSuccess)
    return fail(cuda_fail(cudaGetLastError(), "cudaStreamCreate"));
  const size_t fb = sizeof(float) * p->N;
  if ((st = dalloc(&p->dem, fb)) || (st = dalloc(&p->streams, fb)) ||
      (st = dalloc(&p->noise, fb)) || (st = dalloc(&p->q, fb)) || (st = dalloc(&p->filled, fb)) ||
      (st = dalloc(&p->tmp, fb)) ||
      (st = dalloc(&p->filter, sizeof(float) * (2 * kMaxRunRadius + 1) * (2 * kMaxRunRadius + 1))) ||
      (st = dalloc(&p->code, (size_t)p->N)) || (st = dalloc(&p->dir, 2 * (size_t)p->N)) ||
      (st = dalloc(&p->label, 4 * (size_t)p->N)) ||
      (st = dalloc(&p->counts, 4 * (size_t)p->N)) ||
      (st = dalloc(&p->fill_ws, fill_workspace_bytes(W, H))) ||
      (st = dalloc(&p->route_ws, route_workspace_bytes(W, H))) ||
      (st = dalloc(&p->trace_ws, trace_workspace_bytes(W, H))) ||
      (st = dalloc(&p->dscal, sizeof(uint32_t) * (kRedo + kMaxRedo))))
    return fail(st);
  p->fw = fill_carve(p->fill_ws, W, H);
  p->rw = route_carve(p->route_ws, W, H);
  p->tw = trace_carve(p->trace_ws, W, H);
  cudaStream_t s = p->stream;
#define PCUDA(call)                                          \
  do {                                                       \
    cudaError_t e_ = (call);                                 \
    if (e_ != cudaSuccess) return fail(cuda_fail(e_, #call)); \
  } while (0)
  PCUDA(cudaMemcpyAsync(p->filter, hf.data(), sizeof(float) * taps, cudaMemcpyHostToDevice, s));
  PCUDA(cudaMemcpyAsync(p->dem, dem, fb, kind, s));
  PCUDA(cudaMemcpyAsync(p->streams, streams, fb, kind, s));
  PCUDA(cudaMemsetAsync(p->counts, 0, 4 * (size_t)p->N, s));
  PCUDA(cudaMemsetAsync(p->dscal, 0, sizeof(uint32_t) * kRedo, s));
  // Status words of workspaces that a run may read without having used them
  // (batched steps have workspaces of their own).
  PCUDA(cudaMemsetAsync(p->fw.scal, 0, kFillScalars * sizeof(unsigned int), s));
  PCUDA(cudaMemsetAsync(p->rw.scal, 0, kRouteScalars * sizeof(unsigned int), s));
  PCUDA(cudaMemsetAsync(p->tw.scal, 0, kScalarSlots * sizeof(unsigned int), s));
  {
    // The redo list's place holds the digest until the first realization.
    unsigned long long* dig = (unsigned long long*)(p->dscal + kRedo);
    PCUDA(cudaMemsetAsync(dig, 0, 8, s));
    grid_digest_kernel<<<1024, 256, 0, s>>>(p->dem, p->N, 0x44454dull, dig);
    grid_digest_kernel<<<1024, 256, 0, s>>>(p->streams, p->N, 0x535452ull << 20, dig);
    PCUDA(cudaGetLastError());
    PCUDA(cudaMemcpyAsync(&p->input_digest, dig, 8, cudaMemcpyDeviceToHost, s));
  }
  if ((st = launch_burn_code(p->streams, p->code, W, H, cfg->nodata_stream, cfg->bevel_radius,
                             p->fp.factor, s)))
    return fail(st);
  p->fp.dem = p->dem;
  p->fp.code = p->code;
  p->fp.q = p->q;
  p->fp.min_ord = fill_min_slot(p->fw);
  p->fp.anomaly = (int*)p->dscal + kFlags;
  p->fp.nodata_dem = cfg->nodata_dem;
  p->fp.quantize = cfg->fill_mode == CAGEO_FILL_EXACT ? 0 : 1;
  p->fp.quick = cfg->nodata_dem > 0.0f && cfg->nodata_dem < 4000.0f ? 0 : 1;
  // The front's epilogue sets the fill's seeds.
  p->fp.tseed = p->fw.tseed;
  p->fp.tiles_x = p->fw.tiles_x;
  p->fp.row0 = 0;
  p->fp.W = W;
  p->fp.H = H;
  p->fw.seeded = true;
  p->fw.undone = p->fp.anomaly;
  PCUDA(cudaStreamSynchronize(s));
#undef PCUDA
  *out = p;
  return CAGEO_OK;
}

}  // namespace

extern "C" cageo_status cageo_pipeline_create(cageo_pipeline** out,
                                              const cageo_pipeline_config* cfg,
                                              const float* h_dem, const float* h_streams) {
  return guarded("cageo_pipeline_create", [&] {
    return create_common(out, cfg, h_dem, h_streams, cudaMemcpyHostToDevice);
  });
}

extern "C" cageo_status cageo_pipeline_create_device(cageo_pipeline** out,
                                                     const cageo_pipeline_config* cfg,
                                                     const float* d_dem,
                                                     const float* d_streams) {
  return guarded("cageo_pipeline_create_device", [&] {
    return create_common(out, cfg, d_dem, d_streams, cudaMemcpyDeviceToDevice);
  });
}

// Room for stacks of K realizations.
static cageo_status ensure_stack(cageo_pipeline* p, int K) {
  if (p->stack >= K) return CAGEO_OK;
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  free_stack(p);
  const size_t nb = (size_t)K * p->N;
  cageo_status st;
  if ((st = dalloc(&p->qb, sizeof(float) * nb)) || (st = dalloc(&p->filledb, sizeof(float) * nb)) ||
      (p->N <= kStackNoise && (st = dalloc(&p->noiseb, sizeof(float) * nb))) ||
      (st = dalloc(&p->fill_ws_b, fill_workspace_bytes(p->W, K * p->H))) ||
      (st = dalloc(&p->slab_min, sizeof(unsigned int) * K)) || (st = dalloc(&p->dirb, 2 * nb)) ||
      (st = dalloc(&p->route_ws_b, route_workspace_bytes(p->W, K * p->H))) ||
      (st = dalloc(&p->trace_ws_b, trace_workspace_bytes(p->W, K * p->H)))) {
    free_stack(p);
    cudaGetLastError();
    return st;
  }
  p->stack = K;
  return CAGEO_OK;
}

// The workspaces of a step of K realizations (K <= p->stack), with the single
// fill's tuning.
static void set_step(cageo_pipeline* p, int K) {
  p->step = K;
  p->rwb = route_carve(p->route_ws_b, p->W, K * p->H);
  p->rwb.slab_h = p->H;
  p->twb = trace_carve(p->trace_ws_b, p->W, K * p->H);
  p->twb.slab_h = p->H;
  p->fwb = fill_carve(p->fill_ws_b, p->W, K * p->H);
  p->fwb.slab_h = p->H;
  p->fwb.slab_min = p->slab_min;
  p->fwb.seeded = true;
  p->fwb.wide = p->fw.wide;
  p->fwb.undone = p->fw.undone;
  p->fwb.max_rounds = p->fw.max_rounds;
  p->fwb.flood_warps = p->fw.flood_warps;
}

// Realizations stacked per step where none was asked for.  A realization of a
// small grid is a chain of ~15 launches that leave most of the GPU idle (330
// us at 512^2, 20 of them stacked: 700 us), so as many are stacked as
// make up kStackCells cells (about 32 bytes a cell: 2.1 GB).  Four at 4096^2:
// 3.9 ms in one step, 4.5 in two (6.5 singly, measured with slower stages).
// The limit is one of memory: larger grids gain from stacks, too (8192^2: 3.82 ms a
// realization singly, 3.43 in steps of 4, 3.31 of 16), but at 1.9 GB each a program
// has to ask for those (cageo_pipeline_set_batch).
constexpr int64_t kStackCells = (int64_t)1 << 26;

// Rows of a stack: launches over tiles of 32 rows have them in grid.y.
constexpr int kStackRows = 65535 * 32;

static int stack_of(const cageo_pipeline* p, int count) {
  const int64_t fit = std::min<int64_t>({kMaxStack, kStackCells / p->N, kStackRows / p->H});
  if (p->plain || fit < 2 || count < 2) return 1;
  const int steps = (int)((count + fit - 1) / fit);
  return (count + steps - 1) / steps;  // even steps
}

// Steps start without the wide resolution, whose launch costs 5 us where it is
// not needed (14 us beside other streams' kernels: it asks for room on all SMs).
// A fill that needs it flags its step's realizations, which are then redone like
// those of the burn check; from then on the steps include it.
static void take_wide(cageo_pipeline* p) {
  p->fw.wide = p->fwb.wide = true;
  drop_graph(p);  // captured without it
}

// Waits for a first step (of K realizations) that is about to be captured;
// whether it has to run again with the wide resolution.
static cageo_status first_step_again(cageo_pipeline* p, uint32_t K, bool* again) {
  *again = false;
  if (exact_mode(p) || p->fw.wide) {
    CAGEO_CUDA(cudaStreamSynchronize(p->stream));
    return CAGEO_OK;
  }
  uint32_t scalars[3];  // (the copy to pageable memory waits, too)
  CAGEO_CUDA(cudaMemcpyAsync(scalars, p->dscal, sizeof(scalars), cudaMemcpyDeviceToHost, p->stream));
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  if (!(scalars[kErrors] & kWideSeen)) return CAGEO_OK;
  take_wide(p);
  // Not counted, flagged, listed last: as if it had not run.
  scalars[0] -= K;
  scalars[kErrors] &= kWideSeen - 1u;
  scalars[2] -= K;
  CAGEO_CUDA(cudaMemcpyAsync(p->dscal, scalars, sizeof(scalars), cudaMemcpyHostToDevice, p->stream));
  *again = true;
  return CAGEO_OK;
}

// `steps` stacked steps of K realizations, replaying a captured graph where
// one is wanted: it is captured on first use, and again for another K once
// that has been used by two runs in a row.
static cageo_status run_steps(cageo_pipeline* p, int K, int steps) {
  cudaStream_t s = p->stream;
  cageo_status st;
  if (p->step != K) set_step(p, K);
  int b = 0;
  if (p->cfg.use_graphs && p->graph_k != K && (p->graph_k == 0 || p->last_k == K)) {
    drop_step_graph(p);
    // Warm-up outside capture, then capture one step.
    for (bool again = true; again;) {
      if ((st = enqueue_step(p))) return st;
      if ((st = first_step_again(p, (uint32_t)K, &again))) return st;
    }
    b = 1;
    cudaGraph_t g = nullptr;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      cageo_status cst = enqueue_step(p);
      cudaError_t e = cudaStreamEndCapture(s, &g);
      if (cst != CAGEO_OK || e != cudaSuccess ||
          cudaGraphInstantiate(&p->exec_b, g, 0) != cudaSuccess) {
        p->exec_b = nullptr;
      }
      cudaGetLastError();
    }
    // Kept even when the capture failed: graph_k marks it as tried (steps then
    // run as direct launches).
    p->graph_b = g;
    p->graph_k = K;
  }
  p->last_k = K;
  for (; b < steps; b++) {
    if (p->exec_b && p->graph_k == K) CAGEO_CUDA(cudaGraphLaunch(p->exec_b, s));
    else if ((st = enqueue_step(p))) return st;
  }
  return CAGEO_OK;
}

// At most kMaxRedo realizations, of which any may have to be redone.
static cageo_status run_part(cageo_pipeline* p, uint32_t first, int count) {
  cudaStream_t s = p->stream;
  cageo_status st;
  const uint32_t scalars[kRedo] = {first, 0, 0, first + (uint32_t)count - 1u};
  CAGEO_CUDA(cudaMemcpyAsync(p->dscal, scalars, sizeof(scalars), cudaMemcpyHostToDevice, s));
  const bool stage_only = p->cfg.nodata_dem == 0.0f;
  // Learned warm starts run on the fast path too (never stacked).
  const bool learned = p->ws_params != nullptr && !stage_only;
  int done = 0;
  int64_t fs[kFillStats] = {}, rs[7] = {}, jumps = 0;
  // Stacked steps first: whole ones of the batch asked for, the rest singly;
  // or, sized by the grid, all realizations (the last step may be smaller).
  // All advance the same device counter.
  const bool asked = p->batch > 1;
  int K = stage_only || learned ? 1 : asked ? p->batch : stack_of(p, count);
  if (K > 1 && !asked && ensure_stack(p, K)) {
    p->plain = true;  // no memory for a stack: singly from now on
    K = 1;
  }
  const bool stacked = K > 1 && count >= K;
  if (stacked) {
    const int steps = count / K, tail = asked ? 0 : count - steps * K;
    if ((st = run_steps(p, K, steps))) return st;
    if (tail) {
      set_step(p, tail);
      if ((st = enqueue_step(p))) return st;
    }
    done = steps * K + tail;
  }
  if (count > 0) p->last_batched = stacked && done == count;
  if (!stage_only && count > done && p->cfg.use_graphs && !p->graph_ok && !p->exec) {
    // Warm-up outside capture (kernel attributes, occupancy caches), then
    // capture one realization.
    for (bool again = true; again;) {
      if ((st = enqueue_fast(p))) return st;
      if ((st = first_step_again(p, 1u, &again))) return st;
    }
    done += 1;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      cageo_status cst = enqueue_fast(p);
      cudaGraph_t g = nullptr;
      cudaError_t e = cudaStreamEndCapture(s, &g);
      if (cst == CAGEO_OK && e == cudaSuccess &&
          cudaGraphInstantiate(&p->exec, g, 0) == cudaSuccess) {
        p->graph = g;
        p->graph_ok = true;
      } else {
        if (g) cudaGraphDestroy(g);
        p->exec = nullptr;
      }
      cudaGetLastError();
    }
    // A failed capture leaves the flag off: the launches run directly.
    if (!p->graph_ok) p->cfg.use_graphs = 0;
  }
  for (int i = done; i < count; i++) {
    if (stage_only) {
      if ((st = run_stage_path(p, first + (uint32_t)i))) return st;
    } else if (p->graph_ok) {
      CAGEO_CUDA(cudaGraphLaunch(p->exec, s));
    } else {
      if ((st = enqueue_fast(p))) return st;
    }
  }
  CAGEO_CUDA(cudaStreamSynchronize(s));
  // The last step's status and statistics, then what any step kept.
  const bool top = p->last_batched;
  if ((st = fill_check_status(top ? p->fwb : p->fw, fs))) return st;
  if ((st = route_check_status(top ? p->rwb : p->rw, rs))) return st;
  if ((st = trace_check_status(top ? p->twb : p->tw, &jumps))) return st;
  uint32_t ends[2];  // errors, realizations to redo
  CAGEO_CUDA(cudaMemcpy(ends, p->dscal + kErrors, sizeof(ends), cudaMemcpyDeviceToHost));
  if ((st = kept_status(ends[0]))) return st;
  if ((ends[0] & kWideSeen) && !p->fw.wide) take_wide(p);
  const uint32_t nredo = ends[1];
  if (nredo) {
    std::vector<uint32_t> redo(nredo);
    CAGEO_CUDA(cudaMemcpy(redo.data(), p->dscal + kRedo, sizeof(uint32_t) * nredo,
                          cudaMemcpyDeviceToHost));
    std::sort(redo.begin(), redo.end(),
              [=](uint32_t a, uint32_t b) { return a - first < b - first; });
    for (uint32_t r : redo)
      if ((st = run_stage_path(p, r))) return st;
    CAGEO_CUDA(cudaStreamSynchronize(s));
    if ((st = fill_check_status(p->fw, fs))) return st;
    CAGEO_CUDA(cudaMemcpy(ends, p->dscal + kErrors, sizeof(uint32_t), cudaMemcpyDeviceToHost));
    if ((st = kept_status(ends[0]))) return st;
    p->last_batched = false;  // the last realization computed is the last redone
  }
  p->stats[0] = fs[0];
  p->stats[1] = fs[1];
  p->stats[2] = rs[0];
  p->stats[3] = jumps;
  p->stats[4] = nredo;
  for (int k = 0; k < 9; k++) p->stats[5 + k] = fs[2 + k];
  p->stats[14] = rs[1];
  p->stats[15] = rs[2];
  for (int k = 0; k < 3; k++) p->stats[16 + k] = fs[11 + k];
  for (int k = 0; k < 4; k++) p->stats[19 + k] = rs[3 + k];
  p->stats[23] = fs[14];
  p->stats[24] = fs[15];
  return CAGEO_OK;
}

static cageo_status pipeline_run(cageo_pipeline* p, uint32_t first, int count) {
  CAGEO_CHECK_ARG(p && count >= 0, "pipeline and count");
  // (Whole steps of the batch asked for in every part but the last.)
  const int part = (int)kMaxRedo / p->batch * p->batch;
  for (int64_t redone = 0;;) {
    const int n = std::min(count, part);
    const cageo_status st = run_part(p, first, n);
    if (st) return st;
    p->stats[4] = redone += p->stats[4];
    first += (uint32_t)n;
    count -= n;
    if (count == 0) return CAGEO_OK;
  }
}

extern "C" cageo_status cageo_pipeline_run(cageo_pipeline* p, uint32_t first, int count) {
  return guarded("cageo_pipeline_run", [&] { return pipeline_run(p, first, count); });
}

// One fast-path realization with CUDA events between the stages on the
// pipeline's stream (no graph).  It is a real realization: its border mask
// is accumulated like any other.  h_ms receives up to 6 stage times:
// noise, front (convolution+realistic+burn+quantize), fill, routing,
// tracing, border.
extern "C" cageo_status cageo_pipeline_profile(cageo_pipeline* p, uint32_t realization,
                                               float* h_ms, int n) {
  CAGEO_CHECK_ARG(p && h_ms, "null argument");
  CAGEO_CHECK_ARG(p->cfg.nodata_dem != 0.0f, "profiling needs the fused path (NODATA != 0)");
  cudaStream_t s = p->stream;
  const cageo_pipeline_config& c = p->cfg;
  const WithWide wide(p->fw);
  p->last_batched = false;
  cudaEvent_t ev[7], fm[4];
  for (auto& e : ev) CAGEO_CUDA(cudaEventCreate(&e));
  for (auto& e : fm) CAGEO_CUDA(cudaEventCreate(&e));
  cageo_status st = CAGEO_OK;
  do {
    if (cudaMemcpyAsync(p->dscal, &realization, 4, cudaMemcpyHostToDevice, s) != cudaSuccess) {
      st = cuda_fail(cudaGetLastError(), "cudaMemcpyAsync");
      break;
    }
    if ((st = fill_begin(p->fw, s))) break;
    cudaEventRecord(ev[0], s);
    if ((st = launch_noise(p->noise, p->N, c.seed, 0, p->dscal, c.error_mean, c.error_stddev, s, 1)))
      break;
    cudaEventRecord(ev[1], s);
    if ((st = launch_front(p->noise, p->W, p->H, c.filter_model, p->filter, p->radius, p->fp, s,
                           p->conv_tile, 1)))
      break;
    cudaEventRecord(ev[2], s);
    if (!exact_mode(p)) p->fw.marks = fm;
    st = enqueue_fill(p);
    p->fw.marks = nullptr;
    if (st) break;
    cudaEventRecord(ev[3], s);
    if ((st = enqueue_route(p))) break;
    cudaEventRecord(ev[4], s);
    if ((st = trace_run(p->dir, p->streams, p->code, p->label, p->tw, s, trace_mode(p), false)))
      break;
    cudaEventRecord(ev[5], s);  // the border stage decodes the labels
    if ((st = border_u32_from_state(p->tw, p->label, p->counts, (const int*)p->dscal + kFlags,
                                    trace_mode(p), p->dscal, nullptr, s)))
      break;
    if ((st = enqueue_end(p, step_errors(p->fw, p->rw, p->tw), 1))) break;
    cudaEventRecord(ev[6], s);
    if (cudaStreamSynchronize(s) != cudaSuccess) {
      st = cuda_fail(cudaGetLastError(), "cudaStreamSynchronize");
      break;
    }
    for (int i = 0; i < 6 && i < n; i++) cudaEventElapsedTime(&h_ms[i], ev[i], ev[i + 1]);
    // The fill's parts (CPU-compatible mode): set-up, walled flood, the walls'
    // levels, resolution, and a last part that is empty now.
    const cudaEvent_t fill_marks[6] = {ev[2], fm[0], fm[1], fm[2], fm[3], ev[3]};
    for (int i = 0; i < 5 && 6 + i < n; i++) {
      if (exact_mode(p)) h_ms[6 + i] = 0.0f;
      else cudaEventElapsedTime(&h_ms[6 + i], fill_marks[i], fill_marks[i + 1]);
    }
    int64_t fs[kFillStats], rs[7];
    if ((st = fill_check_status(p->fw, fs))) break;
    p->stats[0] = fs[0];
    p->stats[1] = fs[1];
    for (int k = 0; k < 9; k++) p->stats[5 + k] = fs[2 + k];
    if ((st = route_check_status(p->rw, rs))) break;
    p->stats[2] = rs[0];
    p->stats[14] = rs[1];
    p->stats[15] = rs[2];
    for (int k = 0; k < 3; k++) p->stats[16 + k] = fs[11 + k];
    for (int k = 0; k < 4; k++) p->stats[19 + k] = rs[3 + k];
    p->stats[23] = fs[14];
    p->stats[24] = fs[15];
    st = trace_check_status(p->tw, &p->stats[3]);
  } while (0);
  for (auto& e : ev) cudaEventDestroy(e);
  for (auto& e : fm) cudaEventDestroy(e);
  return st;
}

static cageo_status pipeline_run_filter(cageo_pipeline* p, uint32_t first, int count, int model,
                                        float practical_range, float error_mean,
                                        float error_stddev) {
  CAGEO_CHECK_ARG(p && count >= 0, "pipeline and count");
  CAGEO_CHECK_ARG(model == CAGEO_FILTER_GAUSSIAN || model == CAGEO_FILTER_EXPONENTIAL,
                  "filter model");
  CAGEO_CHECK_ARG(practical_range > 0, "practical range");
  const int r = cageo_filter_radius(practical_range, p->cfg.cell_size);
  CAGEO_CHECK_ARG(r >= 0 && r < p->W && r < p->H && r <= kMaxRunRadius,
                  "filter radius must be below the grid size and 64");
  const int L = 2 * r + 1, taps = model == CAGEO_FILTER_GAUSSIAN ? L : L * L;
  std::vector<float> hf(taps);
  cageo_status st = cageo_filter_build(model, practical_range, p->cfg.cell_size, r, hf.data());
  if (st) return st;
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  CAGEO_CUDA(cudaMemcpy(p->filter, hf.data(), sizeof(float) * taps, cudaMemcpyHostToDevice));
  p->cfg.filter_model = model;
  p->cfg.practical_range = practical_range;
  p->cfg.error_mean = error_mean;
  p->cfg.error_stddev = error_stddev;
  p->radius = r;
  drop_graph(p);  // captured with the old filter's launch shapes
  p->cfg.use_graphs = 0;
  return pipeline_run(p, first, count);
}

extern "C" cageo_status cageo_pipeline_run_filter(cageo_pipeline* p, uint32_t first, int count,
                                                  int model, float practical_range,
                                                  float error_mean, float error_stddev) {
  return guarded("cageo_pipeline_run_filter", [&] {
    return pipeline_run_filter(p, first, count, model, practical_range, error_mean,
                               error_stddev);
  });
}

// Checkpoint file (native byte order): the 8-byte magic "CAGEOCK2", a
// fixed header recording everything the counts depend on -- the grid size,
// the seed, the next realization number, the pipeline's filter and error
// model, bevel radius, fill mode, NODATA values and cell size, and a digest
// of the DEM and stream grids -- then W*H uint32 counts.  Loading refuses a
// checkpoint whose header differs from the pipeline in any of them, so a
// resume can only continue the same Monte Carlo run.
struct CheckpointHeader {
  char magic[8];
  int32_t width, height;
  uint64_t seed;
  uint32_t next_realization;
  int32_t filter_model;
  float practical_range, cell_size, error_mean, error_stddev;
  int32_t bevel_radius, fill_mode;
  float nodata_dem, nodata_stream;
  uint64_t input_digest;
};

static CheckpointHeader checkpoint_header(const cageo_pipeline* p, uint32_t next) {
  CheckpointHeader h;
  std::memset(&h, 0, sizeof(h));
  std::memcpy(h.magic, "CAGEOCK2", 8);
  h.width = p->W;
  h.height = p->H;
  h.seed = p->cfg.seed;
  h.next_realization = next;
  h.filter_model = p->cfg.filter_model;
  h.practical_range = p->cfg.practical_range;
  h.cell_size = p->cfg.cell_size;
  h.error_mean = p->cfg.error_mean;
  h.error_stddev = p->cfg.error_stddev;
  h.bevel_radius = p->cfg.bevel_radius;
  h.fill_mode = p->cfg.fill_mode;
  h.nodata_dem = p->cfg.nodata_dem;
  h.nodata_stream = p->cfg.nodata_stream;
  h.input_digest = p->input_digest;
  return h;
}

// The first header field that differs, or nullptr.  Floats compare by bits.
static const char* checkpoint_mismatch(const CheckpointHeader& a, const CheckpointHeader& b) {
  auto same = [](const void* x, const void* y, size_t n) { return std::memcmp(x, y, n) == 0; };
  if (a.width != b.width || a.height != b.height) return "grid size";
  if (a.seed != b.seed) return "seed";
  if (a.filter_model != b.filter_model) return "filter model";
  if (!same(&a.practical_range, &b.practical_range, 4)) return "practical range";
  if (!same(&a.cell_size, &b.cell_size, 4)) return "cell size";
  if (!same(&a.error_mean, &b.error_mean, 4)) return "error mean";
  if (!same(&a.error_stddev, &b.error_stddev, 4)) return "error standard deviation";
  if (a.bevel_radius != b.bevel_radius) return "bevel radius";
  if (a.fill_mode != b.fill_mode) return "fill mode";
  if (!same(&a.nodata_dem, &b.nodata_dem, 4) || !same(&a.nodata_stream, &b.nodata_stream, 4))
    return "NODATA values";
  if (a.input_digest != b.input_digest) return "DEM or stream grid";
  return nullptr;
}

// The file is written beside the target as "<path>.tmp", flushed to disk and
// renamed over the target, so a crash or kill during the write leaves the
// previous checkpoint intact.
static cageo_status pipeline_save(cageo_pipeline* p, const char* path,
                                  uint32_t next_realization) {
  CAGEO_CHECK_ARG(p && path, "null argument");
  std::vector<uint32_t> h((size_t)p->N);
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  CAGEO_CUDA(cudaMemcpy(h.data(), p->counts, 4 * (size_t)p->N, cudaMemcpyDeviceToHost));
  const std::string tmp = std::string(path) + ".tmp";
  FILE* f = std::fopen(tmp.c_str(), "wb");
  if (!f) {
    set_error("unable to open \"%s\" for writing", tmp.c_str());
    return CAGEO_ERR_IO;
  }
  const CheckpointHeader hd = checkpoint_header(p, next_realization);
  bool ok = std::fwrite(&hd, sizeof(hd), 1, f) == 1 &&
            std::fwrite(h.data(), 4, h.size(), f) == h.size();
  ok = ok && std::fflush(f) == 0 && fsync(fileno(f)) == 0;
  ok = (std::fclose(f) == 0) && ok;
  if (!ok) {
    std::remove(tmp.c_str());
    set_error("short write to \"%s\"", tmp.c_str());
    return CAGEO_ERR_IO;
  }
  if (std::rename(tmp.c_str(), path) != 0) {
    std::remove(tmp.c_str());
    set_error("unable to replace \"%s\"", path);
    return CAGEO_ERR_IO;
  }
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_save(cageo_pipeline* p, const char* path,
                                            uint32_t next_realization) {
  return guarded("cageo_pipeline_save", [&] { return pipeline_save(p, path, next_realization); });
}

static cageo_status pipeline_load(cageo_pipeline* p, const char* path,
                                  uint32_t* next_realization) {
  CAGEO_CHECK_ARG(p && path && next_realization, "null argument");
  FILE* f = std::fopen(path, "rb");
  if (!f) {
    set_error("unable to open checkpoint \"%s\"", path);
    return CAGEO_ERR_IO;
  }
  CheckpointHeader hd;
  std::vector<uint32_t> h((size_t)p->N);
  bool ok = std::fread(&hd, sizeof(hd), 1, f) == 1 && std::memcmp(hd.magic, "CAGEOCK2", 8) == 0;
  if (ok) {
    const CheckpointHeader mine = checkpoint_header(p, hd.next_realization);
    if (const char* what = checkpoint_mismatch(hd, mine)) {
      std::fclose(f);
      set_error("checkpoint \"%s\" belongs to another run (its %s differs)", path, what);
      return CAGEO_ERR_FORMAT;
    }
  }
  ok = ok && std::fread(h.data(), 4, h.size(), f) == h.size() && std::fgetc(f) == EOF;
  std::fclose(f);
  if (!ok) {
    set_error("\"%s\" is not a complete checkpoint", path);
    return CAGEO_ERR_FORMAT;
  }
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  CAGEO_CUDA(cudaMemcpy(p->counts, h.data(), 4 * (size_t)p->N, cudaMemcpyHostToDevice));
  *next_realization = hd.next_realization;
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_load(cageo_pipeline* p, const char* path,
                                            uint32_t* next_realization) {
  return guarded("cageo_pipeline_load", [&] { return pipeline_load(p, path, next_realization); });
}

extern "C" cageo_status cageo_pipeline_counts_device(cageo_pipeline* p, float* d_out) {
  CAGEO_CHECK_ARG(p && d_out, "null argument");
  cageo_status st = counts_to_float(p->counts, d_out, p->N, p->stream);
  if (st) return st;
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_counts(cageo_pipeline* p, float* h_out) {
  CAGEO_CHECK_ARG(p && h_out, "null argument");
  cageo_status st = counts_to_float(p->counts, p->tmp, p->N, p->stream);
  if (st) return st;
  CAGEO_CUDA(cudaMemcpyAsync(h_out, p->tmp, sizeof(float) * p->N, cudaMemcpyDeviceToHost,
                             p->stream));
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_counts_bytes(cageo_pipeline* p, uint8_t* h_out) {
  CAGEO_CHECK_ARG(p && h_out, "null argument");
  cudaStream_t s = p->stream;
  cageo_status st = counts_to_float(p->counts, p->tmp, p->N, s);
  if (st) return st;
  // The byte image is staged in the noise buffer and the min/max pair in the
  // redo list; both are rewritten by the next realization.
  uint8_t* bytes = (uint8_t*)p->noise;
  unsigned int* mm = p->dscal + kRedo;
  if ((st = launch_to_bytes(p->tmp, bytes, p->N, mm, s))) return st;
  CAGEO_CUDA(cudaMemcpyAsync(h_out, bytes, (size_t)p->N, cudaMemcpyDeviceToHost, s));
  CAGEO_CUDA(cudaStreamSynchronize(s));
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_last_stages(cageo_pipeline* p, float* h_filled,
                                                   int8_t* h_dir, int* h_label) {
  CAGEO_CHECK_ARG(p, "null pipeline");
  cudaStream_t s = p->stream;
  // After a stacked step the last realization's filled grid is its top slab.
  const float* filled = p->last_batched ? p->filledb + (size_t)(p->step - 1) * p->N : p->filled;
  if (h_filled)
    CAGEO_CUDA(cudaMemcpyAsync(h_filled, filled, 4 * p->N, cudaMemcpyDeviceToHost, s));
  const int8_t* dir = p->last_batched ? p->dirb + 2 * (size_t)(p->step - 1) * p->N : p->dir;
  if (h_dir) CAGEO_CUDA(cudaMemcpyAsync(h_dir, dir, 2 * p->N, cudaMemcpyDeviceToHost, s));
  if (h_label) CAGEO_CUDA(cudaMemcpyAsync(h_label, p->label, 4 * p->N, cudaMemcpyDeviceToHost, s));
  CAGEO_CUDA(cudaStreamSynchronize(s));
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_reset_counts(cageo_pipeline* p) {
  CAGEO_CHECK_ARG(p, "null pipeline");
  CAGEO_CUDA(cudaMemsetAsync(p->counts, 0, 4 * (size_t)p->N, p->stream));
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  return CAGEO_OK;
}

// Candidate settings of the autotuner: sweep rounds per fill tile visit x
// warps per SM of the fill's flood (with the first convolution
// tile), then the other convolution tiles with the fill setting chosen
// among those (fill fields 0).  The front and the fill are separate stages,
// so tuning them one after the other finds the best of the product.
static const int kTuneRounds[3] = {16, 32, 64};
static const int kTuneWarps[3] = {16, 20, 22};
constexpr int kTuneFill = 9;
constexpr int kTuneCandidates = kTuneFill + kConvTiles - 1;

extern "C" int cageo_autotune_candidates(cageo_tuning* h_out, int n) {
  for (int k = 0; h_out && k < n && k < kTuneCandidates; k++) {
    if (k < kTuneFill) {
      h_out[k] = cageo_tuning{kTuneRounds[k % 3], kTuneWarps[k / 3], 0};
    } else {
      h_out[k] = cageo_tuning{0, 0, k - kTuneFill + 1};
    }
  }
  return kTuneCandidates;
}

// Stacked steps run with the single fill's tuning.
static void sync_step_tuning(cageo_pipeline* p) {
  if (p->step) set_step(p, p->step);
}

extern "C" cageo_status cageo_pipeline_set_tuning(cageo_pipeline* p, const cageo_tuning* t) {
  CAGEO_CHECK_ARG(p && t, "null argument");
  CAGEO_CHECK_ARG(t->fill_rounds >= 1 && t->fill_rounds <= 1024, "fill rounds must be 1..1024");
  CAGEO_CHECK_ARG(fill_flood_warps_valid(t->fill_warps), "fill warps must be 16, 20 or 22");
  CAGEO_CHECK_ARG(t->conv_tile >= 0 && t->conv_tile < kConvTiles,
                  "convolution tile must be 0..3");
  CAGEO_CHECK_ARG(conv_tile_applies(p->cfg.filter_model, p->radius, t->conv_tile),
                  "the convolution tile does not fit this filter radius in shared memory");
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  p->fw.max_rounds = t->fill_rounds;
  p->fw.flood_warps = t->fill_warps;
  p->conv_tile = t->conv_tile;
  sync_step_tuning(p);
  drop_graph(p);  // captured with the old launch shapes
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_get_tuning(cageo_pipeline* p, cageo_tuning* t) {
  CAGEO_CHECK_ARG(p && t, "null argument");
  t->fill_rounds = p->fw.max_rounds;
  t->fill_warps = p->fw.flood_warps;
  t->conv_tile = p->conv_tile;
  return CAGEO_OK;
}

// Autotuning: each candidate runs one warm-up and `trials` realizations on
// the fast path (direct launches, timed with events on the pipeline's
// stream); the fastest is kept and the CUDA graph is captured again on the
// next run.  The counts are reset to zero afterwards.
extern "C" cageo_status cageo_pipeline_autotune(cageo_pipeline* p, uint32_t first, int trials,
                                                cageo_tuning* h_best, float* h_ms, int n_ms) {
  CAGEO_CHECK_ARG(p && trials >= 1, "pipeline and trials");
  CAGEO_CHECK_ARG(p->cfg.nodata_dem != 0.0f && !p->ws_params,
                  "autotuning times the fused path (NODATA != 0, no warm start)");
  cudaStream_t s = p->stream;
  cudaEvent_t e0, e1;
  CAGEO_CUDA(cudaEventCreate(&e0));
  CAGEO_CUDA(cudaEventCreate(&e1));
  cageo_status st = CAGEO_OK;
  const WithWide wide(p->fw);
  p->last_batched = false;
  float best_ms = 0.0f;
  cageo_tuning best{p->fw.max_rounds, p->fw.flood_warps, p->conv_tile};
  cageo_tuning cand[kTuneCandidates];
  cageo_autotune_candidates(cand, kTuneCandidates);
  for (int c = 0; c < kTuneCandidates && st == CAGEO_OK; c++) {
    if (c < kTuneFill) {
      p->fw.max_rounds = cand[c].fill_rounds;
      p->fw.flood_warps = cand[c].fill_warps;
    } else {
      // Another convolution tile with the fill setting chosen above; a tile
      // that does not apply (exponential filters use the 2D kernel) or does
      // not fit the radius is skipped (0 ms).
      cand[c].fill_rounds = best.fill_rounds;
      cand[c].fill_warps = best.fill_warps;
      if (!conv_tile_applies(p->cfg.filter_model, p->radius, cand[c].conv_tile)) {
        if (h_ms && c < n_ms) h_ms[c] = 0.0f;
        continue;
      }
      p->fw.max_rounds = best.fill_rounds;
      p->fw.flood_warps = best.fill_warps;
    }
    p->conv_tile = cand[c].conv_tile;
    const uint32_t r0 = first + (uint32_t)(c * (trials + 1));
    const uint32_t scalars[4] = {r0, 0, 0, r0 + (uint32_t)trials};
    if (cudaMemcpyAsync(p->dscal, scalars, sizeof(scalars), cudaMemcpyHostToDevice, s) !=
        cudaSuccess) {
      st = cuda_fail(cudaGetLastError(), "cudaMemcpyAsync");
      break;
    }
    if ((st = enqueue_fast(p))) break;  // warm-up
    cudaEventRecord(e0, s);
    for (int k = 0; k < trials && st == CAGEO_OK; k++) st = enqueue_fast(p);
    cudaEventRecord(e1, s);
    if (cudaEventSynchronize(e1) != cudaSuccess) {
      st = cuda_fail(cudaGetLastError(), "cudaEventSynchronize");
      break;
    }
    uint32_t kept = 0;
    if (st == CAGEO_OK &&
        cudaMemcpy(&kept, p->dscal + kErrors, sizeof(kept), cudaMemcpyDeviceToHost) != cudaSuccess)
      st = cuda_fail(cudaGetLastError(), "cudaMemcpy");
    if (st == CAGEO_OK) st = kept_status(kept);
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    ms /= (float)trials;
    if (h_ms && c < n_ms) h_ms[c] = ms;
    if (c == 0 || ms < best_ms) {
      best_ms = ms;
      best = cand[c];
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (st) return st;
  p->fw.max_rounds = best.fill_rounds;
  p->fw.flood_warps = best.fill_warps;
  p->conv_tile = best.conv_tile;
  sync_step_tuning(p);
  drop_graph(p);
  if (h_best) *h_best = best;
  CAGEO_CUDA(cudaMemsetAsync(p->counts, 0, 4 * (size_t)p->N, s));
  CAGEO_CUDA(cudaMemsetAsync(p->dscal + 1, 0, (kRedo - 1) * sizeof(uint32_t), s));
  CAGEO_CUDA(cudaStreamSynchronize(s));
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_set_batch(cageo_pipeline* p, int batch) {
  CAGEO_CHECK_ARG(p, "null pipeline");
  CAGEO_CHECK_ARG(batch >= 1 && batch <= kMaxStack, "batch must be 1..64 realizations");
  if (batch > 1) {
    CAGEO_CHECK_ARG(p->cfg.fill_mode == CAGEO_FILL_CPU_COMPAT,
                    "batched steps need the CPU-compatible fill mode");
    CAGEO_CHECK_ARG((int64_t)batch * p->N < kMaxCells, "batch * grid cells must stay below 2^31");
  }
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  free_stack(p);
  p->batch = 1;
  p->plain = batch == 1;
  if (batch == 1) return CAGEO_OK;
  batch = std::min(batch, kStackRows / p->H);  // (at least 32: H <= 65535)
  const cageo_status st = ensure_stack(p, batch);
  if (st) return st;
  set_step(p, batch);
  p->batch = batch;
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_set_warmstart(cageo_pipeline* p, const float* h_params,
                                                     int n, float threshold) {
  CAGEO_CHECK_ARG(p, "null pipeline");
  CAGEO_CUDA(cudaStreamSynchronize(p->stream));
  drop_graph(p);  // the captured step holds the old fill
  if (!h_params) {
    if (p->ws_params) cudaFree(p->ws_params);
    p->ws_params = nullptr;
    return CAGEO_OK;
  }
  CAGEO_CHECK_ARG(p->cfg.fill_mode == CAGEO_FILL_EXACT,
                  "the learned warm start needs the exact fill mode");
  CAGEO_CHECK_ARG(n == cageo_ws_param_count(), "parameter count");
  if (!p->ws_params) CAGEO_CUDA(cudaMalloc((void**)&p->ws_params, sizeof(float) * n));
  if (!p->warm) CAGEO_CUDA(cudaMalloc((void**)&p->warm, sizeof(float) * p->N));
  if (!p->ws_acc) CAGEO_CUDA(cudaMalloc((void**)&p->ws_acc, sizeof(unsigned long long) * 9));
  CAGEO_CUDA(cudaMemcpy(p->ws_params, h_params, sizeof(float) * n, cudaMemcpyHostToDevice));
  CAGEO_CUDA(cudaMemset(p->ws_acc, 0, sizeof(unsigned long long) * 9));
  p->ws_threshold = threshold;
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_warmstart_stats(cageo_pipeline* p, int64_t* h_stats,
                                                       int n) {
  CAGEO_CHECK_ARG(p && h_stats, "null argument");
  unsigned long long acc[9] = {};
  if (p->ws_acc) {
    CAGEO_CUDA(cudaStreamSynchronize(p->stream));
    CAGEO_CUDA(cudaMemcpy(acc, p->ws_acc, sizeof(acc), cudaMemcpyDeviceToHost));
  }
  for (int i = 0; i < n && i < 9; i++) h_stats[i] = (int64_t)acc[i];
  return CAGEO_OK;
}

extern "C" cageo_status cageo_pipeline_graph_kernels(cageo_pipeline* p, int64_t* h_count) {
  CAGEO_CHECK_ARG(p && h_count, "null argument");
  // The stacked step's graph where steps are stacked and it was captured.
  cudaGraph_t g = (p->exec_b && (p->batch > 1 || !p->graph_ok)) ? p->graph_b
                  : (p->graph_ok ? p->graph : nullptr);
  CAGEO_CHECK_ARG(g, "no step has been captured in a CUDA graph");
  size_t n = 0;
  CAGEO_CUDA(cudaGraphGetNodes(g, nullptr, &n));
  std::vector<cudaGraphNode_t> nodes(n);
  CAGEO_CUDA(cudaGraphGetNodes(g, nodes.data(), &n));
  int64_t kernels = 0;
  for (size_t i = 0; i < n; i++) {
    cudaGraphNodeType t;
    CAGEO_CUDA(cudaGraphNodeGetType(nodes[i], &t));
    kernels += t == cudaGraphNodeTypeKernel;
  }
  *h_count = kernels;
  return CAGEO_OK;
}

extern "C" cudaStream_t cageo_pipeline_stream(cageo_pipeline* p) { return p ? p->stream : nullptr; }

extern "C" cageo_status cageo_pipeline_stats(cageo_pipeline* p, int64_t* h_stats, int n) {
  CAGEO_CHECK_ARG(p && h_stats, "null argument");
  for (int i = 0; i < n && i < 25; i++) h_stats[i] = p->stats[i];
  return CAGEO_OK;
}

extern "C" void cageo_pipeline_destroy(cageo_pipeline* p) {
  if (!p) return;
  cudaStreamSynchronize(p->stream);
  free_all(p);
  delete p;
}
