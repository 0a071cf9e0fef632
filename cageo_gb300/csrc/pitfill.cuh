// pitfill.cuh -- CPU-path-compatible pit filling on the GPU (shared with
// pipeline.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "cageo.h"

namespace cageo {

// Workspace of one fill: per-tile states, rims, masks and work queue, and the
// cell lists of the resolution.
struct FillWork {
  int W = 0, H = 0;
  int tiles_x = 0, tiles_y = 0;
  uint8_t* flags = nullptr;      // W*H: cell flags of the resolution
  int* queued = nullptr;         // ntiles: tile state in the work queue (tilequeue.cuh)
  int* lists = nullptr;          // 2 * ntiles + kRingSlack: the work queue's ring
  uint8_t* tseed = nullptr;      // ntiles: tile holds an outlet (or a cell to repair)
  uint8_t* tvis = nullptr;       // ntiles: tile state of the flood (levelflood.cuh)
  uint32_t* cand = nullptr;      // W*H: list of the resolution's cells
  uint32_t* aux = nullptr;       // W*H: their walled level, then component minima (at roots)
  uint32_t* label = nullptr;     // W*H: their component labels
  // The flood (levelflood.cuh), in the space of the labels: per tile the rim
  // entries (4 sides x 32: level bits, flags), and 32 column masks each (lane
  // = column, bit = row) of the cells that are clean, that never relay in
  // the flood, and that are walls (interior and not passable).  (The wide
  // resolution keeps other cells in the first two.)
  uint2* rim = nullptr;
  uint32_t *mclean = nullptr, *mdead = nullptr, *mwall = nullptr;
  unsigned int* scal = nullptr;  // scalar block (see pitfill.cu)
  int max_rounds = 64;           // sweep rounds per tile visit before the tile re-queues itself
  int flood_warps = 20;          // warps per block (per SM) of the flood: 16, 20 or 22
  // Stacked realizations (cold starts of either fill): the grid holds
  // H / slab_h realizations of slab_h rows each, one above the other.
  // Every slab's first and last rows are its border (outlets), so no flood
  // value crosses from one slab to another: a cell that is not on a border
  // has all 8 neighbours in its own slab, and border cells never change.
  // slab_min holds each slab's ordered minimum of q (the passability test's
  // minE).  slab_h = 0: one realization, minimum in the scalar block.
  int slab_h = 0;
  const unsigned int* slab_min = nullptr;
  // The lower bound of the resolution has a budget (see pitfill.cu).  A fill that
  // would exceed it is left to the wide resolution: fill_run launches that, too,
  // if `wide`; if not, such a fill is left unfinished, with undone[k] (not null)
  // set for each slab k, and fill_finish or another fill_run finishes it.
  bool wide = false;
  int* undone = nullptr;
  // The fused front (or fill_quantize_min) has set the tile seeds; otherwise
  // the fill finds them itself.
  bool seeded = false;
  // Profiling only: when set, fill_run records marks[0] after the set-up,
  // [1] after the walled flood, [2] after the walls' levels, [3] after the
  // resolution.
  const cudaEvent_t* marks = nullptr;
};

// Whether `warps` is a block size the flood is built for.
bool fill_flood_warps_valid(int warps);

size_t fill_workspace_bytes(int W, int H);
FillWork fill_carve(void* base, int W, int H);

// First of all: the scalar block, the seeds, the work queue, the tile states
// and the rims of a fill, in one launch.
cageo_status fill_begin(const FillWork& w, cudaStream_t s);
// Fill q (already quantized, min already in scal) into `filled`.  Runs on
// `s`; does not synchronize.  Errors found on the device are reported by
// fill_check_status after the stream has drained.
cageo_status fill_run(const float* q, float* filled, const FillWork& w,
                      float nodata, cudaStream_t s);
// Exact float fill of v (the reference's GPU path): no quantization, no
// minimum needed.  `warm` (may be null): per-cell start values.  The fill
// verifies a warm start itself: after the warm flood, cells whose level no
// chain of relays from an outlet supports restart from +inf and a repair
// flood visits their tiles, so the result is the exact fill for any start.
cageo_status fill_run_exact(const float* v, float* filled, const FillWork& w, float nodata,
                            const float* warm, cudaStream_t s);
// Quantize d in place (the reference's step (i)), reduce its minimum into the
// scalar block and set the tile seeds.
cageo_status fill_quantize_min(float* d, const FillWork& w, float nodata,
                               cudaStream_t s);
unsigned int* fill_min_slot(const FillWork& w);
// Copies the device status (0 ok) and stats into host memory; the stream
// must have been synchronized.  stats (kFillStats entries): last pass
// number, phases, drains of the flood, steps of the lower bound's longest front,
// microseconds of the flood, of the lower bound (of a warm-started exact fill:
// of the repair flood), of the phases, tiles and sweep rounds of the flood,
// tiles and rounds of the repair flood, kilo-cycles summed over tile visits
// spent staging, sweeping, storing, and kilo-cycles warps of the flood and of
// the repair flood spent waiting for a tile, and the cells a warm-started
// exact fill restarted from +inf.
constexpr int kFillStats = 17;
constexpr int kFillScalars = 224;  // words of the scalar block
cageo_status fill_check_status(const FillWork& w, int64_t* stats);
// After a fill_run without `wide`, with the same arguments: waits for it, finishes
// it if it was left unfinished, and checks its status like fill_check_status.
cageo_status fill_finish(const float* q, float* filled, const FillWork& w, float nodata,
                         int64_t* stats, cudaStream_t s);
// The device word that is not 0 after a fill that took, or needs, the wide
// resolution.
const unsigned int* fill_wide_word(const FillWork& w);
// The device word that a fill leaves at 0 or at an error (cleared by the next
// fill_begin), and what that error says.
const unsigned int* fill_error_word(const FillWork& w);
const char* fill_error_text(unsigned int error);
// Adds the last warm-started exact fill's counters to acc (9 device
// uint64: fills, fills that restarted cells, cells restarted, warm-flood
// tile visits and sweep rounds, repair sweep rounds, warm and repair
// microseconds, repair tile visits).  Stream-ordered, no synchronization.
cageo_status fill_accumulate_warm_stats(const FillWork& w, unsigned long long* acc,
                                        cudaStream_t s);

}  // namespace cageo
