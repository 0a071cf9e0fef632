// routing.cuh -- A7 flow routing and A8/A9 tracing and border internals,
// shared with pipeline.cu.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "cageo.h"

namespace cageo {

struct RouteWork {
  int W = 0, H = 0;
  int tiles_x = 0, tiles_y = 0;
  uint8_t* tflat = nullptr;      // per 32x32 tile: holds a flat cell beyond layer 1 (2: visited)
  int* queued = nullptr;         // per tile: state in the work queue
  int* lists = nullptr;          // 2 * ntiles + kRingSlack: the work queue's ring
  uint32_t* mflat = nullptr;     // per tile, 32 row masks (bit = column): flat cells
  uint32_t* mfirst = nullptr;    // the same: flat cells of layer 1
  int* rim = nullptr;            // per tile, 4 sides x 32: distance, 0 where not flat
  unsigned int* scal = nullptr;  // counters, barrier, error
  // Stacked realizations: H / slab_h grids of slab_h rows each, one above
  // the other; each slab's first and last rows are its border (0: one grid).
  // Only the steepest-descent pass needs it: flat cells are interior, so
  // their neighbours lie in their own slab.
  int slab_h = 0;
};
constexpr int kRouteScalars = 224;  // words of the scalar block
size_t route_workspace_bytes(int W, int H);
RouteWork route_carve(void* base, int W, int H);
// mode: CAGEO_ROUTE_CPU_COMPAT or CAGEO_ROUTE_GPU_ORDER (nodata is used by
// the latter only).  flatdist may be null.
cageo_status route_run(const float* filled, int8_t* dir, int* flatdist,
                       const RouteWork& w, cudaStream_t s, int mode, float nodata);
// stats (7 entries, may be null): flat relaxation passes, flat cells,
// microseconds of the flat relaxation, flat tile visits, and kilo-cycles
// summed over visits spent staging, searching, storing.
cageo_status route_check_status(const RouteWork& w, int64_t* stats);
// The device word that a routing leaves at 0 or at an error, and what it says.
const unsigned int* route_error_word(const RouteWork& w);
const char* route_error_text();

struct TraceWork {
  int W = 0, H = 0, tiles_x = 0, tiles_y = 0;
  int* state = nullptr;          // W*H: label, or the tile-border cell the path leaves by
  int* bstate = nullptr;         // 124 per 32x32 tile: the same for the tiles' border cells
  unsigned int* scal = nullptr;
  // Stacked realizations: H / slab_h grids of slab_h rows each, one above the
  // other, over one stream raster of slab_h rows; paths end at their slab's
  // edge (0: one grid).
  int slab_h = 0;
};
size_t trace_workspace_bytes(int W, int H);
TraceWork trace_carve(void* base, int W, int H);
// is_stream(c) = streams[c] >= 0; the label of a stream terminal is
// (int)(-streams[c]).  code (may be null): the burn codes (front.cuh), whose
// stream bit is read instead of the streams.
// mode CAGEO_TRACE_DEAD_END_ERROR: cells whose path ends without an
// outlet are ERROR instead of taking cell 0's label.
// write_labels = false leaves the labels to border_u32_from_state.
cageo_status trace_run(const int8_t* dir, const float* streams, const uint8_t* code, int* label,
                       const TraceWork& w, cudaStream_t s, int mode, bool write_labels);
cageo_status trace_check_status(const TraceWork& w, int64_t* jumps);
// The same for a tracing.
const unsigned int* trace_error_word(const TraceWork& w);
const char* trace_error_text();

// count[i] += border(label) (stage API).
cageo_status border_float(const int* label, float* count, int W, int H,
                          cudaStream_t s);
// From the trace states of a trace_run without labels: adds the border masks
// of all slabs unless *gate is set, and writes the labels (mode as for
// tracing) of slab k where *real + k == *last (last null: of every slab).
cageo_status border_u32_from_state(const TraceWork& w, int* label, uint32_t* count,
                                   const int* gate, int mode, const uint32_t* real,
                                   const uint32_t* last, cudaStream_t s);

}  // namespace cageo
