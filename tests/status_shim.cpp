// status_shim.cpp -- stands in front of a stage's launch function of
// libcageo.so and, after the call a test names, writes an error into the status
// word of that launch, as a stage that reached one of its limits would: an
// error code from a fake of the failing call, with no fault on the GPU.
//
// Loaded into the global scope before libcageo.so, whose calls between its
// source files then bind to the functions below.
#include <dlfcn.h>
#include <cuda_runtime.h>
#include "pitfill.cuh"
#include "routing.cuh"

namespace {
int g_stage, g_call, g_seen;  // 1 fill, 2 routing, 3 tracing; the call of it to fail
void* g_lib;

template <class F>
F* real(F* mine) {
  Dl_info info;
  dladdr((void*)mine, &info);
  return (F*)dlsym(g_lib, info.dli_sname);
}

// Sets the word (zero after a launch that met no limit) to 1 in stream order.
void launched(int stage, const unsigned int* word, cudaStream_t s) {
  if (stage == g_stage && ++g_seen == g_call) cudaMemsetAsync((void*)word, 1, 1, s);
}
}  // namespace

extern "C" void shim_library(const char* path) { g_lib = dlopen(path, RTLD_NOW | RTLD_NOLOAD); }
extern "C" void shim_fail(int stage, int call) {
  g_stage = stage;
  g_call = call;
  g_seen = 0;
}
extern "C" int shim_seen() { return g_seen; }

namespace cageo {
cageo_status fill_run(const float* q, float* filled, const FillWork& w, float nodata,
                      cudaStream_t s) {
  const cageo_status st = real(fill_run)(q, filled, w, nodata, s);
  launched(1, w.scal + 3, s);
  return st;
}
cageo_status route_run(const float* filled, int8_t* dir, int* flatdist, const RouteWork& w,
                       cudaStream_t s, int mode, float nodata) {
  const cageo_status st = real(route_run)(filled, dir, flatdist, w, s, mode, nodata);
  launched(2, w.scal + 3, s);
  return st;
}
cageo_status trace_run(const int8_t* dir, const float* streams, const uint8_t* code, int* label,
                       const TraceWork& w, cudaStream_t s, int mode, bool write_labels) {
  const cageo_status st = real(trace_run)(dir, streams, code, label, w, s, mode, write_labels);
  launched(3, w.scal + 2, s);
  return st;
}
}  // namespace cageo
