// pitfill.cu -- A6 pit filling with the semantics of the reference's CPU
// path (src/pitfilling/PitFillingAlgorithmCPUOpenMP.h:68-242), and the exact
// float fill of its GPU path (src/pitfilling/PitFillingAlgorithmGPUCUDA.cu:
// 201-381) as a second mode: the flood alone on the unquantized grid, every
// outlet relaying, unreached cells ending at the GPU path's 99990000.
//
// The CPU fill is a bucket priority-flood over 1 mm levels in which a
// popped cell expands its neighbours only if its value v survives
// toElev(toIndex(v)) == v ("passable").  The result is: outlets (border
// cells and cells equal to 0) keep q; every other reached cell gets
// W = max(q, L) where L is the lowest value among neighbours that expand;
// a non-passable cell expands only when it was reached at a level L >= q;
// unreached cells keep q.  Whether a non-passable cell expands depends only
// on cells with a strictly lower q, so the solution is unique, and it is
// computed here by monotone relaxations:
//
//   1. walled flood: only passable cells relay.  Every level is a path the
//      reference's fill may take, so the result S is an upper bound; a
//      non-passable cell with S == q was reached below q (its incoming level
//      is a passable value, never q itself) and is a wall for good.  On
//      terrain rounded to 1 mm about 1% of the cells are non-passable, and S
//      differs from the answer on 0.1-0.2% of the cells: pockets of lakes cut
//      off by non-passable cells under water (S > q), which do expand.
//   2. lower bound A: from S, the non-passable cells with S > q relay as well
//      (and go on relaying when they fall below q): the cells that truly
//      expand are among them, so A <= answer <= S.  If no such cell ends at
//      or below its q, A solves the fill's equation, whose solution is
//      unique: A is the answer.
//   3. otherwise the cells with A != S form 8-connected components that no
//      change can leave.  A component without a cell of the kind just named
//      is settled at A.  In the others the cells restart at S, those
//      non-passable cells with A > q are confirmed (they certainly expand),
//      and the levels relax to an upper bound B.  Where B == A both are the
//      answer.  The cells between A and B form components of their own, for
//      which phases follow: M = the component's least level among unconfirmed
//      non-passable cells above their q; every such cell with q <= M is
//      confirmed (no later change can take its level below M); relax; until
//      none is left.
//
// Steps 2 and 3 work on lists of cells (fill_resolve_kernel), or, where the
// lower bound would take long that way, on tiles again
// (fill_resolve_wide_kernel); the flood of
// step 1 -- and the exact fill, which is that flood without walls -- is a
// persistent cooperative kernel over 32x32 tiles (levelflood.cuh): one warp
// owns a tile at a time and sweeps it until it is a fixed point for its
// neighbours' rims; a tile whose rim changed queues the neighbouring tiles on
// an asynchronous work queue (no pass barriers; tilequeue.cuh).  The flood
// ends when no tile is queued or in process.  Every wait and every loop is
// bounded; exceeding a bound sets an error flag that the host turns into
// CAGEO_ERR_NO_CONVERGENCE.
#include <algorithm>
#include "common.cuh"
#include "fillflags.cuh"
#include "levelflood.cuh"
#include "pitfill.cuh"
#include "stage_math.cuh"
#include "tilequeue.cuh"

namespace cageo {

// Scalar block layout (unsigned ints).
enum : int {
  S_MIN = 0,       // ordered min of q (minE)
  S_ERR = 3,       // 0 ok; 1 barrier wait; 2 idle wait; 3 queue state; 4 visits; 5 phases; 6 union
  S_RESULT = 8,    // resolution: whether a thread passed true to the last barrier
  S_MORE_AT = 9,   // S_MORE at the last barrier
  S_CAND = 10,     // walls on the list of the resolution
  S_MORE = 22,     // cells listed by the resolution itself
  S_OPEN = 23,     // cells of the reopened components
  S_UNSURE = 24,   // walls between the bounds A and B
  S_FRONT = 25,    // other cells among the first S_UNSURE of the list
  S_BEHIND = 26,   // such walls after those
  S_WIDE = 27,     // 1: the lower bound is left to the wide resolution
  S_PASS = 11,     // floods and relaxations run so far in this fill
  S_PHASES = 12,
  S_PASSES_A = 13, // drains of the flood (1)
  S_STEPS = 14,    // relaxation steps of the resolution's longest front, before the phases
  S_US_A = 15,     // microseconds of the flood
  S_US_B = 16,     // microseconds of the lower bound (or of a repair flood)
  S_US_P = 17,     // microseconds of the phases
  S_RESET = 21,    // warm-started exact fill: cells restarted from +inf (unsupported)
  // Per-visit statistics, updated by every tile visit: a line of their own
  // (96..127), away from the error flag that idle warps poll.
  S_TILES_A = 96,   // tiles processed by the flood
  S_ROUNDS_A = 97,  // sweep rounds run by the flood
  S_TILES_B = 98,   // tiles processed by a repair flood
  S_ROUNDS_B = 99,  // sweep rounds run by a repair flood
  S_KCYC_LOAD = 100,   // kilo-cycles (summed over tile visits) staging tiles
  S_KCYC_SWEEP = 101,  // kilo-cycles sweeping
  S_KCYC_STORE = 102,  // kilo-cycles writing back and queueing
  S_KCYC_IDLE_A = 103, // kilo-cycles warps of the flood waited for a tile (tail included)
  S_KCYC_IDLE_B = 104, // the same for a repair flood
  S_HEAD = 128,      // work-queue tickets handed out (own 128-byte line)
  S_TAIL = 160,      // work-queue entries pushed (own line)
  S_DONE = 192,      // tiles finished (own line)
  S_BAR_COUNT = kBarCountSlot,
  S_BAR_GEN = kBarGenSlot,
  S_SIZE = kFillScalars
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Per-cell flag bits of the resolution.
constexpr unsigned int kActive = 1, kConfirmed = 2, kMember = 4, kReopened = 8, kUnsure = 16,
                       kUnsureWall = 32;

// The space that the flood's rims and masks share with the component labels
// of the resolution: the labels are the larger part except on grids only a
// few cells wide.
static size_t shared_bytes(size_t n, size_t nt) {
  return std::max(align_up(n * 4, 256), align_up(nt * kRimCells * sizeof(uint2), 256) +
                                            3 * align_up(nt * kTile * 4, 256));
}

size_t fill_workspace_bytes(int W, int H) {
  size_t n = (size_t)W * H;
  size_t nt = (size_t)((W + kTile - 1) / kTile) * ((H + kTile - 1) / kTile);
  return align_up(n, 256) + align_up(nt * 4, 256) + align_up((2 * nt + kRingSlack) * 4, 256) +
         2 * align_up(nt, 256) + 2 * align_up(n * 4, 256) + shared_bytes(n, nt) + 1024;
}

FillWork fill_carve(void* base, int W, int H) {
  FillWork w;
  w.W = W;
  w.H = H;
  w.tiles_x = (W + kTile - 1) / kTile;
  w.tiles_y = (H + kTile - 1) / kTile;
  size_t n = (size_t)W * H, nt = (size_t)w.tiles_x * w.tiles_y;
  char* p = (char*)base;
  w.flags = (uint8_t*)p;
  p += align_up(n, 256);
  w.queued = (int*)p;
  p += align_up(nt * 4, 256);
  w.lists = (int*)p;
  p += align_up((2 * nt + kRingSlack) * 4, 256);
  w.tseed = (uint8_t*)p;
  p += align_up(nt, 256);
  w.tvis = (uint8_t*)p;
  p += align_up(nt, 256);
  w.aux = (uint32_t*)p;
  p += align_up(n * 4, 256);
  w.cand = (uint32_t*)p;
  p += align_up(n * 4, 256);
  w.label = (uint32_t*)p;
  char* r = p;
  w.rim = (uint2*)r;
  r += align_up(nt * kRimCells * sizeof(uint2), 256);
  w.mclean = (uint32_t*)r;
  r += align_up(nt * kTile * 4, 256);
  w.mdead = (uint32_t*)r;
  r += align_up(nt * kTile * 4, 256);
  w.mwall = (uint32_t*)r;
  p += shared_bytes(n, nt);
  w.scal = (unsigned int*)p;
  return w;
}

unsigned int* fill_min_slot(const FillWork& w) { return w.scal + S_MIN; }

// ---- asynchronous tile work queue (tilequeue.cuh) --------------------------
// The fill's queue: tile states in w.queued, the ring in w.lists
// (2 * ntiles + kRingSlack slots), counters in the scalar block.
__device__ __forceinline__ TileQueue fill_queue(const FillWork& w) {
  return TileQueue{w.queued,
                   w.lists,
                   2u * (unsigned int)(w.tiles_x * w.tiles_y) + kRingSlack,
                   w.scal + S_HEAD,
                   w.scal + S_TAIL,
                   w.scal + S_DONE,
                   (int*)(w.scal + S_ERR)};
}

__device__ __forceinline__ void flush_stats(const FillWork& w, VisitStats& st, bool b_slots) {
  if (!st.tiles && !st.kidle) return;
  atomicAdd(&w.scal[b_slots ? S_TILES_B : S_TILES_A], st.tiles);
  atomicAdd(&w.scal[b_slots ? S_ROUNDS_B : S_ROUNDS_A], st.rounds);
  atomicAdd(&w.scal[S_KCYC_LOAD], st.kload);
  atomicAdd(&w.scal[S_KCYC_SWEEP], st.ksweep);
  atomicAdd(&w.scal[S_KCYC_STORE], st.kstore);
  if (st.kidle) atomicAdd(&w.scal[b_slots ? S_KCYC_IDLE_B : S_KCYC_IDLE_A], st.kidle);
  st = VisitStats{};
}

// Lock-free union-find over the cells of the resolution (w.label): links
// always point to a smaller cell index, so no cycle can form; roots are
// hooked with CAS, paths halved with plain stores.  Bounded loops.
// The root without path halving: the flattening pass writes each cell's
// root while other threads walk the same paths, and a halving store that
// landed after such a write would replace the root by an ancestor below
// it -- leaving a cell labelled with a non-root, outside its component's
// minimum.  Plain reads only, so every store of that pass is a root.
__device__ __forceinline__ uint32_t uf_root(const uint32_t* lab, uint32_t x) {
  for (int it = 0; it < (1 << 20); it++) {
    const uint32_t p = ((const volatile uint32_t*)lab)[x];
    if (p == x) return x;
    x = p;
  }
  return x;
}

// Both paths are climbed at once, so a step's two reads overlap.
__device__ __forceinline__ bool uf_unite(uint32_t* lab, uint32_t a, uint32_t b) {
  volatile uint32_t* l = lab;
  for (int it = 0; it < (1 << 20); it++) {
    if (a == b) return true;
    const uint32_t pa = l[a], pb = l[b];
    if (pa == a && pb == b) {
      const uint32_t lo = min(a, b), hi = max(a, b);
      if (atomicCAS(&lab[hi], hi, lo) == hi) return true;
      continue;
    }
    // Two steps up where there are two; the cell passed points there, too.
    const uint32_t ga = l[pa], gb = l[pb];
    if (ga != pa) lab[a] = ga;
    if (gb != pb) lab[b] = gb;
    a = ga;
    b = gb;
  }
  return false;
}

// One warp: process queued tiles (visit(t, stats)) until no tile is queued or
// being processed anywhere; a ticket still waiting then is abandoned (head,
// tail and done are reset after the drain).  b_slots: the statistics go to the
// repair flood's counters.  False on an error or a wait limit.
template <class Visit>
__device__ bool drain(const FillWork& w, int lane, int ntiles, bool b_slots, Visit visit) {
  volatile unsigned int* vs = w.scal;
  const unsigned int visit_cap = 1000u * (unsigned int)min(ntiles, 4000000);
  const TileQueue q = fill_queue(w);
  long long ticket = -1;
  unsigned int ns = 32, finished = 0;
  VisitStats st;
  bool ok = true;
  long long idle_from = -1;  // clock when this warp last found no tile (-1: busy)
  for (long long idle = 0;;) {
    int t = -1;
    if (lane == 0) t = tq_try_dequeue(q, &ticket);
    t = __shfl_sync(0xffffffffu, t, 0);
    __syncwarp();  // lane 0's fence holds for the loads of all lanes (a shuffle orders no memory)
    if (t >= 0) {
      if (lane == 0 && idle_from >= 0) st.kidle += (unsigned int)((clock64() - idle_from) >> 10);
      idle_from = -1;
      visit(t, st);
      if (lane == 0) {
        tq_finish(q, t);
        finished++;
        if (st.tiles >= 64) flush_stats(w, st, b_slots);
      }
      __syncwarp();
      idle = 0;
      ns = 32;
      continue;
    }
    int end = 0;  // 1 drained, 2 error, 3 limit
    if (lane == 0) {
      if (tq_drained(q, &finished)) end = 1;
      else if (vs[S_ERR]) end = 2;
      else if (idle > (1LL << 25)) end = 3;
      else if (vs[b_slots ? S_TILES_B : S_TILES_A] > visit_cap) end = 4;
    }
    end = __shfl_sync(0xffffffffu, end, 0);
    if (end) {
      ok = end == 1;
      if (lane == 0 && end > 2) atomicCAS((int*)(w.scal + S_ERR), 0, end == 3 ? 2 : 4);
      break;
    }
    idle++;
    if (idle_from < 0) idle_from = clock64();
    __nanosleep(ns);
    if (ns < 512) ns <<= 1;
  }
  if (lane == 0) {
    if (idle_from >= 0) st.kidle += (unsigned int)((clock64() - idle_from) >> 10);
    flush_stats(w, st, b_slots);
  }
  __syncwarp();
  return ok;
}

// Seed the queue with the marked tiles (a tile without an outlet, or without
// a cell to repair, cannot change before a neighbour does, which queues it),
// one 2x2 parity class of tiles after another with a grid barrier in
// between, so the ring holds them class by class.  Tiles taken at the same
// time are then rarely neighbours, and each class starts from the finished
// borders of the classes before it: in a CPU simulation of the queue (2048^2
// realization, 1/29 of the tiles in flight) this took the visits per tile
// from 3.19 in plain tile order to 2.68.
__device__ __forceinline__ bool seed_queue(const FillWork& w, const GridSync& gs, int gwarp,
                                           int nwarps, int lane, int ntiles) {
  bool go = true;
  const TileQueue q = fill_queue(w);
  for (int c = 0; c < 4 && go; c++) {
    for (int base = gwarp * 32; base < ntiles; base += nwarps * 32) {
      const int i = base + lane, tx = i % w.tiles_x, ty = i / w.tiles_x;
      tq_enqueue(q, i < ntiles && ((tx & 1) | ((ty & 1) << 1)) == c && w.tseed[i], i);
    }
    go = grid_barrier(gs, gridDim.x);
  }
  return go;
}

// The walled flood, the exact fill (no walls), the warm-started exact fill
// (MARKS: with clean marks) and its repair flood.  Blocks of at most WARPS
// warps, one per SM; a small grid's tiles are spread over all SMs with fewer
// warps each.
template <bool MARKS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) level_flood_kernel(LevelArgs a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  LevelSmem& s = reinterpret_cast<LevelSmem*>(smraw)[warp];
  const FillWork& w = a.w;
  const int gwarp = blockIdx.x * warps + warp, nwarps = gridDim.x * warps;
  const int ntiles = w.tiles_x * w.tiles_y;
  GridSync gs{w.scal + S_BAR_COUNT, w.scal + S_BAR_GEN, (int*)(w.scal + S_ERR)};
  const unsigned long long t_start = global_ns();
  bool go = seed_queue(w, gs, gwarp, nwarps, lane, ntiles);
  const bool repair = a.stage == 3;
  if (go)
    go = drain(w, lane, ntiles, repair, [&](int t, VisitStats& st) {
      level_visit<MARKS>(s, a, fill_queue(w), t, lane, st);
    });
  grid_barrier(gs, gridDim.x);
  // Tiles no outlet reaches were never queued: their masks and start levels
  // are written here, so that every tile holds them.
  for (int t = gwarp; t < ntiles && !repair; t += nwarps)
    if (__ldcg(w.tvis + t) == 0) level_untouched(a, t, lane);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    volatile unsigned int* vs = w.scal;
    vs[S_PASS] = vs[S_PASS] + 2;
    const unsigned int us = (unsigned int)((global_ns() - t_start) / 1000);
    if (!repair) vs[S_PASSES_A] = 1;
    vs[repair ? S_US_B : S_US_A] = us;
  }
}

// Start of a fill: the scalar block, the seeds, the tile states, the work
// queue (no tile queued, the ring empty), the rims (no level, no flag) and the
// cell flags, in
// one launch instead of a kernel and six memsets (2 us each).
__global__ void fill_begin_kernel(FillWork w, int ntiles) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = tid; i < S_SIZE; i += nthreads)
    w.scal[i] = i == S_MIN ? 0xffffffffu : 0u;
  const int64_t ring = 2 * (int64_t)ntiles + kRingSlack;
  for (int64_t i = tid; i < ring; i += nthreads) {
    w.lists[i] = kEmptySlot;
    if (i < ntiles) {
      w.queued[i] = kIdle;
      w.tseed[i] = 0;
      w.tvis[i] = 0;
    }
  }
  const uint4 none = make_uint4(0x7f800000u, 0u, 0x7f800000u, 0u);  // two entries (+inf, 0)
  uint4* rim = reinterpret_cast<uint4*>(w.rim);
  for (int64_t i = tid; i < (int64_t)ntiles * (kRimCells / 2); i += nthreads) rim[i] = none;
  uint4* f = reinterpret_cast<uint4*>(w.flags);  // (its space is a multiple of 256 bytes)
  const int64_t fw = ((int64_t)w.W * w.H + 15) / 16;
  for (int64_t i = tid; i < fw; i += nthreads) f[i] = make_uint4(0u, 0u, 0u, 0u);
}

// The seeds of a grid no other kernel has marked: tiles holding an outlet (a
// border cell of its slab, or a cell at 0).  One warp per tile.
__global__ void __launch_bounds__(256) fill_seed_kernel(const float* __restrict__ q, FillWork w) {
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= w.tiles_x * w.tiles_y) return;
  const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
  const int slab_h = w.slab_h ? w.slab_h : w.H;
  bool any = false;
#pragma unroll 8
  for (int y = y0; y < y0 + kTile; y++) {
    if (x >= w.W || y >= w.H) break;
    const int ys = y % slab_h;
    any |= x == 0 || x == w.W - 1 || ys == 0 || ys == slab_h - 1 ||
           q[(int64_t)y * w.W + x] == 0.0f;
  }
  if (__any_sync(0xffffffffu, any) && lane == 0) w.tseed[t] = 1;
}

// A warm start is no lower than the elevation.
__global__ void fill_warm_start_kernel(const float* __restrict__ v, const float* __restrict__ warm,
                                       float* __restrict__ Wg, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) Wg[i] = fmaxf(warm[i], v[i]);
}

// Verification of a warm-started exact fill.  The warm flood keeps clean
// marks: in exact mode every reached cell relays, so a marked cell's level
// is supported -- a chain of relays from an outlet reaches it with no step
// above its level -- and such a level is never below the exact fill (the
// chain is a path whose highest elevation it covers).  At the flood's
// fixpoint no cell is above the exact fill either (induction along its
// optimal path), so a supported cell holds the answer.  Every other cell
// (started too low, pulled down by one that was, or unreached) restarts
// from +inf, in the grid and in its tile's rim, and marks its tile for the
// repair flood; with every start an upper bound again, the repair flood ends
// at the exact fill.  One warp per tile.  Also resets the work queue's
// positions.
__global__ void __launch_bounds__(256) fill_unsupported_kernel(LevelArgs a) {
  const FillWork& w = a.w;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    w.scal[S_HEAD] = 0u;
    w.scal[S_TAIL] = 0u;
    w.scal[S_DONE] = 0u;
  }
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= w.tiles_x * w.tiles_y) return;
  // Every tile was visited (a warm start seeds them all).
  const unsigned int reset = ~(w.mdead[t * kTile + lane] | w.mclean[t * kTile + lane]);
  const bool any = __any_sync(0xffffffffu, reset != 0);
  if (lane == 0) w.tseed[t] = any;
  if (!any) return;
  float* wp = a.Wg + (int64_t)(t / w.tiles_x) * kTile * w.W + (t % w.tiles_x) * kTile + lane;
  for (int y = 0; y < kTile; y++)
    if ((reset >> y) & 1u) wp[(int64_t)y * w.W] = kInf;
  uint2* rim = w.rim + (size_t)t * kRimCells + lane;
  const uint2 none = make_uint2(0x7f800000u, 0u);
  if (reset & 1u) rim[kTop * kTile] = none;
  if (reset >> 31) rim[kBottom * kTile] = none;
  const unsigned int l = __shfl_sync(0xffffffffu, reset, 0), r = __shfl_sync(0xffffffffu, reset, 31);
  if ((l >> lane) & 1u) rim[kLeft * kTile] = none;
  if ((r >> lane) & 1u) rim[kRight * kTile] = none;
  const unsigned int n = __reduce_add_sync(0xffffffffu, (unsigned int)__popc(reset));
  if (lane == 0) {
    w.tvis[t] = kVisited | kUnsettled;
    atomicAdd(&w.scal[S_RESET], n);
  }
}

// Cells no outlet reaches keep the reference's initial value: only tiles that
// hold one are touched.  One warp per tile.
__global__ void __launch_bounds__(256) fill_final_exact_kernel(LevelArgs a) {
  const FillWork& w = a.w;
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= w.tiles_x * w.tiles_y || !(w.tvis[t] & kUnreached)) return;
  const unsigned int dead = w.mdead[t * kTile + lane];
  float* wp = a.Wg + (int64_t)(t / w.tiles_x) * kTile * w.W + (t % w.tiles_x) * kTile + lane;
  for (int y = 0; y < kTile; y++) {
    if ((dead >> y) & 1u) continue;  // (cells outside the grid among them)
    if (wp[(int64_t)y * w.W] == kInf) wp[(int64_t)y * w.W] = 99990000.0f;
  }
}

// Whether a cell relays by its own nature: passable and not NODATA.
__device__ __forceinline__ bool relays(float q, float minE, float nodata) {
  return q != nodata && passable_quantized(q, minE);
}

// After the walled flood: the levels of the walls (interior non-passable
// cells), W = max(q, least relay of the 8 neighbours), and the list of those
// above their q, which the resolution starts from.  Walls are about 1% of the
// cells, so the pass reads their masks (0.125 B a cell) and gathers each
// wall's 8 neighbours.  The levels of listed walls are left marked (see the
// resolution).  One warp per tile.
__global__ void __launch_bounds__(256) fill_walls_kernel(LevelArgs a) {
  const FillWork& w = a.w;
  const int t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (t >= w.tiles_x * w.tiles_y) return;
  unsigned int wall = w.mwall[t * kTile + lane];
  const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
  const int slab_h = w.slab_h ? w.slab_h : w.H;
  bool unreached = false;
  while (__any_sync(0xffffffffu, wall != 0)) {
    bool lake = false;
    int64_t i = 0;
    if (wall) {
      const int y = y0 + __ffs(wall) - 1;
      wall &= wall - 1;
      i = (int64_t)y * w.W + x;
      const float minE = ordered_to_float(a.minslot[y / slab_h]);
      const float qv = a.q[i];
      float m = kInf;
#pragma unroll
      for (int k = 0; k < 8; k++) {  // a wall is interior: all 8 are in its slab
        const int64_t n = i + (int64_t)d8_dy(k) * w.W + d8_dx(k);
        const float qn = a.q[n], wn = a.Wg[n];
        if (relays(qn, minE, a.nodata)) m = fminf(m, wn);
      }
      const float lv = fmaxf(qv, m);
      lake = lv > qv && lv < kInf;
      a.Wg[i] = lake ? -lv : lv;
      unreached |= lv == kInf;
      if (lake) {
        w.flags[i] = kActive;
        w.aux[i] = __float_as_uint(lv);
      }
    }
    const unsigned int ball = __ballot_sync(0xffffffffu, lake);
    unsigned int base = 0;
    if (lane == 0 && ball) base = atomicAdd(&w.scal[S_CAND], (unsigned int)__popc(ball));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (lake) w.cand[base + __popc(ball & ((1u << lane) - 1u))] = (uint32_t)i;
  }
  if (__any_sync(0xffffffffu, unreached) && lane == 0) w.tvis[t] |= kUnreached;
}

// ---- resolution (steps 2 and 3 of the header) --------------------------------
// Cells are listed once (cand) with the walled flood's level S in aux.  Levels
// are >= 0 here (quantized elevations), so a float's bits order like the
// float, and its sign is free: it marks the level of a listed cell, for the
// length of the resolution.  A fall is one atomicMin of the marked level as a
// signed integer: marked levels are below every unmarked one and ordered
// among themselves, and the first to lower a cell gets S back, unmarked.  The
// other flags are bytes changed by atomics on the word around them.
struct Resolve {
  const float* q;
  float* Wg;
  FillWork w;
  float nodata;
  const unsigned int* minslot;
  int slab_h;

  __device__ __forceinline__ unsigned int* word(int64_t c) const {
    return reinterpret_cast<unsigned int*>(w.flags) + (c >> 2);
  }
  __device__ __forceinline__ unsigned int set(int64_t c, unsigned int f) const {
    const int sh = (int)(c & 3) * 8;
    return (atomicOr(word(c), f << sh) >> sh) & 0xffu;
  }
  __device__ __forceinline__ void clear(int64_t c, unsigned int f) const {
    atomicAnd(word(c), ~(f << ((int)(c & 3) * 8)));
  }
  __device__ __forceinline__ unsigned int get(int64_t c) const {
    return (__ldcg(word(c)) >> ((int)(c & 3) * 8)) & 0xffu;
  }
  // Level of a cell that is not NODATA, and whether it is listed.
  __device__ __forceinline__ float level(int64_t c, bool* listed = nullptr) const {
    const float v = __ldcg(Wg + c);
    if (listed) *listed = __float_as_int(v) < 0;
    return fabsf(v);
  }
  __device__ __forceinline__ float walled(int64_t c) const {  // S of a listed cell
    return __uint_as_float(__ldcg(w.aux + c));
  }
  __device__ __forceinline__ bool wall(int64_t c, float qv) const {
    const int slab = (int)(c / w.W) / slab_h;
    return !passable_quantized(qv, ordered_to_float(minslot[slab]));
  }
};

// Two blocks on an SM: a step's few cells leave most of a block waiting (batch
// 8 at 8192^2: 27.1 ms; one block of 1024 28.1; four of 256 27.5, and slower on
// long lists of few fronts).
constexpr int kResolveThreads = 512;
// Entries of the list a block takes at a time at most (walls; cells of reopened
// components), and entries per block of the launch: with 1024 a block (one
// on a grid of 512x512) the passes over the list took several turns each.
constexpr unsigned int kResolveRun = 512, kReopenRun = 256, kResolveShare = 128;
constexpr int kFrontCells = 1024, kFreshCells = 2048;

// A block's front: cells whose level fell (or walls that have come to relay),
// with that level; one buffer is read while the other fills.  Three counters
// in turn, so a step needs one block barrier.
struct Front {
  uint32_t cell[2][kFrontCells];
  float level[2][kFrontCells];
  int n[3];
  int full;  // an entry did not fit: its cell was marked kActive instead
  int stop;  // a block has left the lower bound to the wide resolution
  // Cells to list.  They are listed many at a time: an addition to the list's
  // length in every step made it three dependent L2 accesses instead of two.
  uint32_t fresh[kFreshCells];
  int nfresh;
  unsigned int at;
  unsigned int gen;  // grid barriers passed (thread 0)
};

// Grid barrier of the `nblocks` blocks of the resolution.  Returns whether any
// thread passed true; *more = the entries listed by then (nothing is listed
// between the last arrival, which takes the number, and the release); f.stop =
// whether the fill is left to the wide resolution; *ok = false on an error (any
// block's) or a wait limit.
__device__ bool any_of(const FillWork& w, Front& f, unsigned int nblocks, bool mine,
                       unsigned int* more, bool* ok) {
  __shared__ unsigned int sh_any, sh_more, sh_ok;
  volatile unsigned int* vs = w.scal;
  const int block = __syncthreads_or(mine);
  if (threadIdx.x == 0) {
    __threadfence();
    sh_ok = 1u;
    if (nblocks == 1) {
      sh_any = block ? 1u : 0u;
      sh_more = vs[S_MORE] | vs[S_WIDE] << 31;
    } else {
      // (The generation is counted, not read here: a read could be performed
      // after the arrival, and after the release that it is to wait for.)
      const unsigned int gen = f.gen++;
      // The count of the arrivals, and 65536 times that of those with a true.
      const unsigned int arrived = atomicAdd(&w.scal[S_BAR_COUNT], block ? 65537u : 1u);
      if ((arrived & 0xffffu) == nblocks - 1) {
        vs[S_BAR_COUNT] = 0u;
        vs[S_RESULT] = block || arrived >> 16 ? 1u : 0u;
        vs[S_MORE_AT] = vs[S_MORE] | vs[S_WIDE] << 31;  // (S_MORE is below 2^31)
        __threadfence();
        atomicAdd(&w.scal[S_BAR_GEN], 1u);
      } else {
        unsigned int ns = 32;
        long long polls = 0;
        while (vs[S_BAR_GEN] == gen) {
          if (++polls > 20000000LL) {  // several seconds
            atomicCAS((int*)(w.scal + S_ERR), 0, 1);
            break;
          }
          if ((polls & 63) == 0 && vs[S_ERR]) break;
          __nanosleep(ns);
          if (ns < 256) ns <<= 1;
        }
      }
      __threadfence();
      sh_any = vs[S_RESULT];
      sh_more = vs[S_MORE_AT];
    }
    if (vs[S_ERR]) sh_ok = 0u;
    f.stop = (int)(sh_more >> 31);
  }
  __syncthreads();
  const bool any = sh_any != 0u;
  *more = sh_more & 0x7fffffffu;
  *ok = sh_ok != 0u;
  __syncthreads();
  return any && *ok;
}

// The whole block: lists the fresh cells from entry `end` + S_MORE on.
__device__ void list_fresh(const Resolve& r, Front& f, unsigned int end) {
  __syncthreads();
  const int n = min(f.nfresh, kFreshCells);
  if (n == 0) return;
  if (threadIdx.x == 0) f.at = atomicAdd(&r.w.scal[S_MORE], (unsigned int)n);
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) __stcg(r.w.cand + end + f.at + i, f.fresh[i]);
  __syncthreads();
  if (threadIdx.x == 0) f.nfresh = 0;
  __syncthreads();
}

__device__ __forceinline__ void front_push(const Resolve& r, Front& f, int buf, int cnt, uint32_t c,
                                           float lv) {
  const int pos = atomicAdd(&f.n[cnt], 1);
  if (pos < kFrontCells) {
    f.cell[buf][pos] = c;
    f.level[buf][pos] = lv;
  } else {
    __threadfence();  // the level before the mark
    r.set(c, kActive);
    f.full = 1;
  }
}

// The whole block: follows its front (buffer 0, f.n[0] entries) until no level
// falls.  THREADS: the block's, 0: any number.  LOWER: `work` counts entries, and
// 128 for each step (64 take ~0.5 us); past the budget, or where another block's
// is spent, the rest is left to the wide resolution: returns whether it is.
template <bool LOWER, int THREADS>
__device__ __forceinline__ bool follow(const Resolve& r, Front& f, unsigned int nu0,
                                       unsigned int budget, unsigned int& steps, unsigned int& work) {
  const FillWork& w = r.w;
  volatile unsigned int* vs = w.scal;
  int buf = 0, cnt = 0;
  bool stop = false;  // (thread 0's)
  for (;;) {
    // (A half full buffer is emptied; what does not fit a step is listed at once.)
    if (__syncthreads_or(LOWER && threadIdx.x == 0 && (f.nfresh > kFreshCells / 2 || stop))) {
      if (threadIdx.x == 0) f.stop = stop;
      list_fresh(r, f, nu0);  // (a block barrier at least)
      if (f.stop) return true;
    }
    const int nf = min(f.n[cnt], kFrontCells);
    const int nxt = cnt == 2 ? 0 : cnt + 1;
    if (threadIdx.x == 0) f.n[nxt == 2 ? 0 : nxt + 1] = 0;
    if (nf == 0) return false;
    if (++steps > (1u << 26)) {  // every step lowers a level: far beyond any path
      if (threadIdx.x == 0) atomicCAS((int*)(w.scal + S_ERR), 0, 4);
      return false;
    }
    if (LOWER && threadIdx.x == 0) {
      const unsigned int before = work;
      work += 128u + (unsigned int)nf;
      if (work > budget) {
        vs[S_WIDE] = 1u;
        stop = true;
      } else if ((work ^ before) & 8192u) {  // (a look costs the block an L2 access)
        stop = vs[S_WIDE] != 0u;
      }
    }
    const int k = threadIdx.x & 7;
    for (int e = threadIdx.x >> 3; e < nf; e += (THREADS ? THREADS : (int)blockDim.x) / 8) {
      const uint32_t c = f.cell[buf][e];
      const float lv = f.level[buf][e];
      const int nx = (int)(c % (uint32_t)w.W) + d8_dx(k), ny = (int)(c / (uint32_t)w.W) + d8_dy(k);
      if (nx < 0 || nx >= w.W || ny < 0 || ny >= w.H) continue;
      const int64_t b = (int64_t)ny * w.W + nx;
      const float qb = r.q[b], nv = fmaxf(qb, lv);
      const unsigned int fl = LOWER ? 0u : r.get(b);  // (kConfirmed does not change meanwhile)
      // (Outlets are at their elevation.)
      if (!(nv < r.level(b)) || qb == r.nodata) continue;
      const int mine = (int)(__float_as_uint(nv) | 0x80000000u);
      const int prev = atomicMin(reinterpret_cast<int*>(r.Wg + b), mine);
      if (LOWER) {
        const bool first = prev >= 0;
        const unsigned int at = warp_append((unsigned int*)&f.nfresh, first);
        if (first) {
          __stcg(w.aux + b, (unsigned int)prev);
          __stcg(w.label + b, (uint32_t)b);
          if (at < kFreshCells) f.fresh[at] = (uint32_t)b;
          else __stcg(w.cand + nu0 + atomicAdd(&w.scal[S_MORE], 1u), (uint32_t)b);
        }
      }
      if (prev <= mine) continue;
      // A wall that falls was above its q, so LOWER lets it relay.
      if (LOWER || !r.wall(b, qb) || ((fl & kConfirmed) && nv > qb))
        front_push(r, f, buf ^ 1, nxt, (uint32_t)b, nv);
    }
    buf ^= 1;
    cnt = nxt;
  }
}

// Relaxes from the active cells among the first nl of a list -- after that, what
// a full buffer left among all na of it -- until no level falls.
// LOWER: the list is cand; walls with S > q relay whatever their level, and a
// neighbour that falls is listed (from entry nu0 on, *more of them so far);
// otherwise the list holds the reopened components or the cells between the
// bounds, confirmed walls above their q relay, and only these cells can fall.
// minima: the least pending levels (aux) of the first nl cells' components are
// reset.
//
// The falls travel up to ~70 cells at 4096^2 (~170 at 8192^2) from where they
// start, so what counts is the time of a step.  Each block follows the fronts
// of its own entries with no grid barrier in between: 8 lanes per cell, one
// per neighbour, two dependent L2 accesses (the neighbour's level and
// elevation, the atomicMin) and one block barrier a step (1.2 us; 1.6 with the
// list's length raised in every step).  Levels fall in any
// order, and a cell two blocks reach is followed by whichever lowers it.
// (Grid-wide rounds over the list took 3.3 ms at 8192^2, a flag beside each
// level -- two accesses more a step -- 0.7 ms.)  Blocks take runs of
// consecutive entries, which lie in the same tiles.
template <bool LOWER>
__device__ unsigned int relax(const Resolve& r, Front& f, const uint32_t* list, unsigned int nl,
                              unsigned int na, unsigned int nblocks, bool minima,
                              unsigned int* more, bool* ok, unsigned int budget = 0) {
  const FillWork& w = r.w;
  const unsigned int nu0 = nl;
  unsigned int steps = 0, work = 0;
  bool again_all = false, stop = false;
  for (bool again = true; again; again_all = true) {
    const unsigned int nu = LOWER ? nl + *more : again_all ? na : nl;
    const unsigned int run = min(LOWER ? kResolveRun : kReopenRun, (nu + nblocks - 1) / nblocks);
    if (threadIdx.x == 0) f.full = f.nfresh = 0;
    for (unsigned int base = blockIdx.x * run; base < nu && !stop; base += nblocks * run) {
      __syncthreads();
      if (threadIdx.x < 3) f.n[threadIdx.x] = 0;
      __syncthreads();
      // The active entries that can lower a neighbour.
      static_assert(kResolveRun <= kResolveThreads && kReopenRun <= kResolveThreads, "one a thread");
      const unsigned int j = base + threadIdx.x;
      for (bool once = j < min(nu, base + run); once; once = false) {
        const uint32_t c = __ldcg(list + j);
        const unsigned int fl = r.get(c);
        if (LOWER) {
          if (j < nu0) w.label[c] = c;
        } else if (minima && !again_all) {
          __stcg(w.aux + __ldcg(w.label + c), 0xffffffffu);
        }
        if (!(fl & kActive)) continue;
        r.clear(c, kActive);
        __threadfence();  // a fall after the read below marks the cell again
        const float lv = r.level(c), qc = r.q[c];
        // (LOWER: every active cell is a wall with S > q, or fell, or both.)
        if (!LOWER && r.wall(c, qc) && !((fl & kConfirmed) && lv > qc)) continue;
        const int x = (int)(c % (uint32_t)w.W), y = (int)(c / (uint32_t)w.W);
        bool lowers = false;
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int nx = x + d8_dx(k), ny = y + d8_dy(k);
          if (nx < 0 || nx >= w.W || ny < 0 || ny >= w.H) continue;
          const int64_t b = (int64_t)ny * w.W + nx;
          const float qb = r.q[b];
          lowers |= fmaxf(qb, lv) < r.level(b) && qb != r.nodata;
        }
        if (lowers) front_push(r, f, 0, 0, c, lv);
      }
      stop = follow<LOWER, kResolveThreads>(r, f, nu0, budget, steps, work);
    }
    if (LOWER) list_fresh(r, f, nu0);
    __syncthreads();
    again = any_of(w, f, nblocks, f.full != 0, more, ok);
    if (LOWER && f.stop) again = false;  // (in every block)
  }
  return steps;
}

// Work (follow()) that a block may spend on the lower bound: about the time that
// the wide resolution's floods take, 0.3 ms and 45 ns per 1000 cells, so at worst
// a fill takes twice as long as by the better way.  Terrain with streams stays far
// below it: the longest front takes 157 steps of at most 2986 at 8192^2, 425 of
// 11178 on 16384^2 cells with lakes, 178 of 508 on 2016x3073 with lakes.
__device__ __forceinline__ unsigned int wide_budget(const FillWork& w) {
  return 32768u + (unsigned int)((int64_t)w.W * w.H / 192);
}

// Steps 2 and 3, and the cells no outlet reaches.  A cooperative launch; only
// as many blocks as the list's runs need stay (a barrier among few blocks is
// cheap, and the list is short on small grids).
__global__ void __launch_bounds__(kResolveThreads, 2) fill_resolve_kernel(Resolve r) {
  __shared__ Front front;
  const FillWork& w = r.w;
  volatile unsigned int* vs = w.scal;
  const unsigned int nu0 = vs[S_CAND];  // (final before the launch)
  const unsigned int nblocks = min(gridDim.x, max(1u, (nu0 + kResolveShare - 1) / kResolveShare));
  if (blockIdx.x >= nblocks) return;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nthreads = (int64_t)nblocks * blockDim.x;
  if (threadIdx.x == 0) front.gen = vs[S_BAR_GEN];  // (any_of fences before it arrives)
  const unsigned long long t0 = global_ns();
  int phases = 0;
  unsigned int more = 0;
  bool ok = true;
  if (nu0) {
    const unsigned int steps =
        relax<true>(r, front, w.cand, nu0, 0u, nblocks, false, &more, &ok, wide_budget(w));
    if (threadIdx.x == 0) atomicMax(&w.scal[S_STEPS], steps);
    if (front.stop) {
      if (tid == 0) vs[S_US_B] = (unsigned int)((global_ns() - t0) / 1000);
      if (w.undone && !w.wide)
        for (int64_t k = tid; k < w.H / r.slab_h; k += nthreads) w.undone[k] = 1;
      return;
    }
  }
  const unsigned long long t1 = global_ns();
  const unsigned int nu = ok ? nu0 + more : 0u;
  // Members: the cells between the bounds, united with their W, NW, N and NE
  // neighbours among them (each pair once).  Reopened components: those with
  // a wall that S left above its q and A took to it.
  bool reopen = false, united = true;
  // Four threads a cell, one per neighbour.  (Their levels first: most
  // neighbours are not listed.)
  for (int64_t j = tid; j < 4 * (int64_t)nu; j += nthreads) {
    const int d = (int)(j & 3);
    const uint32_t c = __ldcg(w.cand + (j >> 2));
    const int cx = (int)(c % (uint32_t)w.W), cy = (int)(c / (uint32_t)w.W);
    const int nx = cx + (d == 0 ? -1 : d - 2), ny = cy + (d == 0 ? 0 : -1);
    const bool in = nx >= 0 && ny >= 0 && nx < w.W;
    const uint32_t b = in ? (uint32_t)ny * (uint32_t)w.W + (uint32_t)nx : c;
    bool lb;
    const float wc = r.level(c), wb = r.level(b, &lb);
    const float qc = r.q[c], sc = r.walled(c);
    if (wc == sc || qc == r.nodata) continue;  // not a member
    if (d == 0) {
      r.set(c, kMember);
      reopen |= wc <= qc && sc > qc && r.wall(c, qc);
    }
    if (!in || !lb) continue;
    const float qb = r.q[b], sb = r.walled(b);
    if (wb != sb && qb != r.nodata) united &= uf_unite(w.label, c, b);
  }
  if (!united) atomicCAS((int*)(w.scal + S_ERR), 0, 6);
  if (nu0 && any_of(w, front, nblocks, reopen, &more, &ok)) {
    for (int64_t j = tid; j < nu; j += nthreads) {
      const uint32_t c = __ldcg(w.cand + j);
      if (!(r.get(c) & kMember)) continue;
      const uint32_t root = uf_root(w.label, c);
      w.label[c] = root;
      const float qc = r.q[c];
      if (r.level(c) <= qc && r.walled(c) > qc && r.wall(c, qc)) r.set(root, kReopened);
    }
    any_of(w, front, nblocks, false, &more, &ok);
    // The cells of reopened components restart at S -- or at what a settled
    // listed wall beside them offers, if that is less -- with the walls that A
    // left above their q confirmed, and are listed once more after the others
    // (where the list fills the array, it is used whole).  aux holds their A
    // from here on.
    const bool apart = 2 * (uint64_t)nu <= (uint64_t)w.W * w.H;
    for (int64_t j = tid; j < nu && ok; j += nthreads) {
      const uint32_t c = __ldcg(w.cand + j);
      if (!(r.get(c) & kMember)) continue;
      const uint32_t root = __ldcg(w.label + c);
      // Every label is a root: a cell labelled otherwise would miss its
      // component's mark.
      if (__ldcg(w.label + root) != root) atomicCAS((int*)(w.scal + S_ERR), 0, 6);
      const bool open = r.get(root) & kReopened;
      if (open) {
        const float qc = r.q[c], lv = r.level(c), s = r.walled(c);
        float start = s;
        const int x = (int)(c % (uint32_t)w.W), y = (int)(c / (uint32_t)w.W);
        unsigned int near = 0;  // the listed neighbours
        float lb[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int nx = x + d8_dx(k), ny = y + d8_dy(k);
          if (nx < 0 || nx >= w.W || ny < 0 || ny >= w.H) continue;
          bool listed;
          lb[k] = r.level((int64_t)ny * w.W + nx, &listed);
          if (listed) near |= 1u << k;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) {
          if (!(near >> k & 1u)) continue;
          const int64_t b = (int64_t)(y + d8_dy(k)) * w.W + x + d8_dx(k);
          const float qb = r.q[b];
          if (lb[k] > qb && qb != r.nodata && !(r.get(b) & kMember) && r.wall(b, qb))
            start = fminf(start, fmaxf(qc, lb[k]));
        }
        const bool confirm = lv > qc && s > qc && r.wall(c, qc);
        if (confirm || start < s) r.set(c, (confirm ? kConfirmed : 0u) | kActive);
        __stcg(w.aux + c, __float_as_uint(lv));
        __stcg(r.Wg + c, -start);
      }
      const unsigned int pos = warp_append(&w.scal[S_OPEN], open && apart);
      if (open && apart) __stcg(w.cand + nu + pos, c);
    }
    any_of(w, front, nblocks, false, &more, &ok);
    const unsigned int no = apart ? vs[S_OPEN] : nu;
    uint32_t* list = apart ? w.cand + nu : w.cand;
    if (ok) relax<false>(r, front, list, no, no, nblocks, false, &more, &ok);
    // The upper bound B; the cells above A are labelled anew.
    auto between = [&](uint32_t c) { return (r.get(c) & kUnsure) != 0; };
    bool unsure = false;
    for (int64_t j = tid; j < no && ok; j += nthreads) {
      const uint32_t c = __ldcg(list + j);
      const bool u = (r.get(c) & kMember) &&
                     (apart || (r.get(__ldcg(w.label + c)) & kReopened)) && r.level(c) != r.walled(c);
      const bool wall = u && r.wall(c, r.q[c]);
      warp_append(&w.scal[S_UNSURE], wall);
      if (!u) continue;
      r.set(c, kUnsure | (wall ? kUnsureWall : 0u));
      __stcg(w.label + c, c);
      unsure |= wall;
    }
    if (any_of(w, front, nblocks, unsure, &more, &ok)) {
      // The walls among them, which are all that the phases look at, move to the
      // front of the list, in exchange for others (whose places are noted in
      // aux, which is free now; at most half of the list each).
      const unsigned int nq = vs[S_UNSURE];
      uint32_t *places = w.aux, *behind = w.aux + (uint64_t)w.W * w.H / 2;
      bool joined = true;
      for (int64_t j = tid; j < no; j += nthreads) {
        const uint32_t c = __ldcg(list + j);
        const unsigned int f = r.get(c);
        const bool u = f & kUnsureWall;
        const unsigned int a = warp_append(&w.scal[S_FRONT], !u && j < nq);
        const unsigned int b = warp_append(&w.scal[S_BEHIND], u && j >= nq);
        if (!u && j < nq) __stcg(places + a, (uint32_t)j);
        if (u && j >= nq) __stcg(behind + b, (uint32_t)j);
        if (!(f & kUnsure)) continue;
        const int cx = (int)(c % (uint32_t)w.W), cy = (int)(c / (uint32_t)w.W);
#pragma unroll 1
        for (int d = 0; d < 4; d++) {  // W, NW, N, NE
          const int nx = cx + (d == 0 ? -1 : d - 2), ny = cy + (d == 0 ? 0 : -1);
          if (nx < 0 || ny < 0 || nx >= w.W) continue;
          const uint32_t n = (uint32_t)ny * (uint32_t)w.W + (uint32_t)nx;
          if (between(n)) joined &= uf_unite(w.label, c, n);
        }
      }
      if (!joined) atomicCAS((int*)(w.scal + S_ERR), 0, 6);
      any_of(w, front, nblocks, false, &more, &ok);
      const unsigned int moves = vs[S_FRONT];
      for (int64_t k = tid; k < moves && ok; k += nthreads) {
        const uint32_t a = __ldcg(places + k), b = __ldcg(behind + k);
        const uint32_t ca = __ldcg(list + a), cb = __ldcg(list + b);
        __stcg(list + a, cb);
        __stcg(list + b, ca);
      }
      any_of(w, front, nblocks, false, &more, &ok);
      // From here aux holds the components' least pending level (at their roots).
      for (int64_t j = tid; j < nq && ok; j += nthreads) {
        const uint32_t c = __ldcg(list + j), root = uf_root(w.label, c);
        w.label[c] = root;
        __stcg(w.aux + root, 0xffffffffu);
      }
      any_of(w, front, nblocks, false, &more, &ok);
      while (ok) {
        // The unconfirmed walls above their q.
        auto pending = [&](int64_t j, uint32_t& c, float& lv, float& qc) {
          c = __ldcg(list + j);
          if (r.get(c) & kConfirmed) return false;
          qc = r.q[c];
          lv = r.level(c);
          return lv > qc;
        };
        bool some = false;
        uint32_t c;
        float lv, qc;
        for (int64_t j = tid; j < nq; j += nthreads) {
          if (!pending(j, c, lv, qc) || lv == kInf) continue;
          const uint32_t root = __ldcg(w.label + c);
          // Every label is a root: a cell labelled otherwise would take a minimum
          // nothing resets.
          if (phases == 0 && __ldcg(w.label + root) != root)
            atomicCAS((int*)(w.scal + S_ERR), 0, 6);
          atomicMin(&w.aux[root], __float_as_uint(lv));
          some = true;
        }
        if (!any_of(w, front, nblocks, some, &more, &ok)) break;
        // Each phase confirms at least one cell of every component with a
        // pending one (the cell holding its minimum).
        if (++phases > (int)min(nq, 0x7fffff00u) + 8) {
          if (threadIdx.x == 0) atomicCAS((int*)(w.scal + S_ERR), 0, 5);
          break;  // (in every block)
        }
        for (int64_t j = tid; j < nq; j += nthreads) {
          if (!pending(j, c, lv, qc)) continue;
          const unsigned int m = __ldcg(w.aux + __ldcg(w.label + c));
          if (m != 0xffffffffu && qc <= __uint_as_float(m)) r.set(c, kConfirmed | kActive);
        }
        any_of(w, front, nblocks, false, &more, &ok);
        if (ok) relax<false>(r, front, list, nq, no, nblocks, true, &more, &ok);
      }
    }
  }
  // The marks come off, and cells no outlet reached keep q.
  for (int64_t j = tid; j < nu0 + more; j += nthreads) {
    const uint32_t c = __ldcg(w.cand + j);
    const float lv = r.level(c);
    r.Wg[c] = lv == kInf ? r.q[c] : lv;
  }
  // (Only tiles that held one after the flood are read.  One warp per tile.)
  const int ntiles = w.tiles_x * w.tiles_y, lane = threadIdx.x & 31;
  for (int64_t t = tid >> 5; t < ntiles; t += nthreads >> 5) {
    if (!(w.tvis[t] & kUnreached)) continue;
    const int x = (int)(t % w.tiles_x) * kTile + lane, y0 = (int)(t / w.tiles_x) * kTile;
    for (int y = y0; y < min(y0 + kTile, w.H) && x < w.W; y++) {
      const int64_t i = (int64_t)y * w.W + x;
      if (r.level(i) == kInf) r.Wg[i] = r.q[i];
    }
  }
  if (tid == 0) {
    vs[S_PASS] = vs[S_PASS] + 1u + (unsigned int)phases;
    vs[S_PHASES] = (unsigned int)phases;
    vs[S_US_B] = (unsigned int)((t1 - t0) / 1000);
    vs[S_US_P] = (unsigned int)((global_ns() - t1) / 1000);
  }
}

// ---- wide resolution ---------------------------------------------------------
// Terrain without streams has lakes whose level the walls under water decide
// far and wide: the falls of the lower bound then reach most cells, many times
// over, and following them cell by cell takes longer than any flood.  The
// resolution above gives up such a fill (S_WIDE), and this kernel, which leaves
// at once otherwise, takes it from there: both bounds by floods over tiles
// (levelflood.cuh), the cells between them listed tile by tile, and phases that
// look at the walls still pending only, with every SM (the resolution above has
// blocks for the list it starts from).  Whole fills, in ms, by the lists alone
// and so: rough ground of 512^2 cells 38 and 13, of 2048^2 824 and 106; hills of
// 2048^2 804 and 257, of 5000x3001 147 and 26; a bowl of 1024^2 11.9 and 1.9.
// Bound by the phases: 0.05 to 0.3 ms each, of which there are up to 2000, and
// in them by the fronts of lakes that drain one after another.
//
// The floods use the tiles' rims and masks, in the space of the labels; mdead
// holds the cells that do not relay in the present flood, mclean the walls that
// the walled flood left above their q (up), of which the second flood's start
// keeps those not confirmed.

// Levels of tile t's rim, from this lane's column: level(y), or +inf where dead.
template <class Level, class Elev>
__device__ __forceinline__ void wide_rim(const FillWork& w, int t, int lane, unsigned int dead,
                                         Level level, Elev elev) {
  uint2* rim = w.rim + (size_t)t * kRimCells;
  for (int y = 0; y < kTile; y++) {
    const bool d = (dead >> y) & 1u;
    const float v = d ? kInf : level(y);
    const uint2 e = make_uint2(__float_as_uint(v), d || v == elev(y) ? kRimFinal : 0u);
    if (y == 0) rim[kTop * kTile + lane] = e;
    if (y == kTile - 1) rim[kBottom * kTile + lane] = e;
    if (lane == 0) rim[kLeft * kTile + y] = e;
    if (lane == kTile - 1) rim[kRight * kTile + y] = e;
  }
}

// Start of the lower bound's flood: the levels so far without their marks (they
// are no lower than the bound), S of every cell in aux.
__device__ __forceinline__ void wide_start_lower(const LevelArgs& a, int t, int lane) {
  const FillWork& w = a.w;
  const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
  const int64_t base = (int64_t)y0 * w.W + x;
  const CellMasks m =
      cell_masks(w, a.minslot, a.nodata, x, y0, [&](int y) { return a.q[base + (int64_t)y * w.W]; });
  const unsigned int never = m.dead & ~m.wall;
  unsigned int up = 0;
  for (int y = 0; y < kTile; y++) {
    if ((never >> y) & 1u) continue;
    const int64_t i = base + (int64_t)y * w.W;
    const float v = a.Wg[i];
    float s = v;
    if (__float_as_int(v) < 0) {  // listed: S is in aux
      s = __uint_as_float(w.aux[i]);
      a.Wg[i] = fabsf(v);
    } else {
      w.aux[i] = __float_as_uint(v);
    }
    if (((m.wall >> y) & 1u) && s > a.q[i]) up |= 1u << y;
  }
  const unsigned int dead = m.dead & ~up;
  w.mdead[t * kTile + lane] = dead;
  w.mwall[t * kTile + lane] = m.wall;
  w.mclean[t * kTile + lane] = up;
  wide_rim(w, t, lane, dead, [&](int y) { return __ldcg(a.Wg + base + (int64_t)y * w.W); },
           [&](int y) { return a.q[base + (int64_t)y * w.W]; });
  if (lane == 0) {
    w.tvis[t] = kVisited | kUnsettled;
    w.tseed[t] = 1;
  }
}

// Start of the upper bound's flood: levels at S, A in aux, the walls that A
// left above their q confirmed.  Only tiles with A != S can change.
__device__ __forceinline__ void wide_start_upper(const LevelArgs& a, int t, int lane) {
  const FillWork& w = a.w;
  const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
  const int64_t base = (int64_t)y0 * w.W + x;
  const unsigned int wall = w.mwall[t * kTile + lane], up = w.mclean[t * kTile + lane];
  const unsigned int all = w.mdead[t * kTile + lane] | up, never = all & ~wall;
  unsigned int confirmed = 0;
  bool fell = false;
  for (int y = 0; y < kTile; y++) {
    if (x >= w.W || y0 + y >= w.H) break;
    const int64_t i = base + (int64_t)y * w.W;
    bool sure = false;
    if (!((never >> y) & 1u)) {
      const float v = __ldcg(a.Wg + i), s = __uint_as_float(w.aux[i]);
      if (v != s) {
        a.Wg[i] = s;
        w.aux[i] = __float_as_uint(v);
        fell = true;
      }
      sure = ((up >> y) & 1u) && v > a.q[i];
    }
    if (sure) confirmed |= 1u << y;
    w.flags[i] = sure ? kConfirmed : 0;
  }
  const unsigned int dead = all & ~confirmed;
  w.mdead[t * kTile + lane] = dead;
  w.mclean[t * kTile + lane] = up & ~confirmed;
  wide_rim(w, t, lane, dead, [&](int y) { return __ldcg(a.Wg + base + (int64_t)y * w.W); },
           [&](int y) { return a.q[base + (int64_t)y * w.W]; });
  fell = __any_sync(0xffffffffu, fell);
  if (lane == 0) {
    w.tvis[t] = kVisited | kUnsettled;
    w.tseed[t] = fell;
  }
}

// Upper bound of the walls not confirmed: they do not relay.
__device__ __forceinline__ void wide_walls(const Resolve& r, int t, int lane) {
  const FillWork& w = r.w;
  const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
  for (unsigned int m = w.mclean[t * kTile + lane]; m; m &= m - 1) {
    const int y = y0 + __ffs(m) - 1;
    const int64_t i = (int64_t)y * w.W + x;
    const float minE = ordered_to_float(r.minslot[y / r.slab_h]);
    float least = kInf;
#pragma unroll
    for (int k = 0; k < 8; k++) {  // a wall is interior: all 8 are in its slab
      const int64_t n = i + (int64_t)d8_dy(k) * w.W + d8_dx(k);
      if (relays(r.q[n], minE, r.nodata) || (r.get(n) & kConfirmed))
        least = fminf(least, __ldcg(r.Wg + n));
    }
    const float v = fmaxf(r.q[i], least);
    if (v < __ldcg(r.Wg + i)) __stcg(r.Wg + i, v);
  }
}

// The cells of tile t where the bounds differ are flagged, the walls not
// confirmed among them counted.
__device__ __forceinline__ void wide_between(const Resolve& r, int t, int lane) {
  const FillWork& w = r.w;
  const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
  const unsigned int never = w.mdead[t * kTile + lane] & ~w.mwall[t * kTile + lane];
  const unsigned int open = w.mclean[t * kTile + lane];
  unsigned int walls = 0;
  for (int y = 0; y < kTile && x < w.W && y0 + y < w.H; y++) {
    if ((never >> y) & 1u) continue;
    const int64_t i = (int64_t)(y0 + y) * w.W + x;
    if (__ldcg(r.Wg + i) == r.walled(i)) continue;
    const bool is_wall = (open >> y) & 1u;
    w.flags[i] |= kUnsure | (is_wall ? kUnsureWall : 0u);  // (this lane's byte)
    walls += is_wall;
  }
  walls = __reduce_add_sync(0xffffffffu, walls);
  if (lane == 0 && walls) atomicAdd(&w.scal[S_UNSURE], walls);
}

// Those cells listed: such walls from the list's start, others from nq on, row by row.
__device__ __forceinline__ void wide_list(const Resolve& r, int t, int lane, unsigned int nq) {
  const FillWork& w = r.w;
  const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
  unsigned int any = 0, wall = 0;
  for (int y = 0; y < kTile && x < w.W && y0 + y < w.H; y++) {
    const unsigned int f = __ldcg(w.flags + (int64_t)(y0 + y) * w.W + x);
    if (f & kUnsure) any |= 1u << y;
    if (f & kUnsureWall) wall |= 1u << y;
  }
  const unsigned int all = __reduce_add_sync(0xffffffffu, (unsigned int)__popc(any));
  if (!all) return;
  const unsigned int walls = __reduce_add_sync(0xffffffffu, (unsigned int)__popc(wall));
  unsigned int at = 0, other = 0;
  if (lane == 0) {
    at = atomicAdd(&w.scal[S_FRONT], walls);
    other = nq + atomicAdd(&w.scal[S_BEHIND], all - walls);
  }
  at = __shfl_sync(0xffffffffu, at, 0);
  other = __shfl_sync(0xffffffffu, other, 0);
  for (int y = 0; y < kTile; y++) {
    const bool u = (any >> y) & 1u, is_wall = (wall >> y) & 1u;
    const unsigned int bw = __ballot_sync(0xffffffffu, is_wall);
    const unsigned int bo = __ballot_sync(0xffffffffu, u && !is_wall);
    const unsigned int below = (1u << lane) - 1u;
    if (u) {
      const int64_t i = (int64_t)(y0 + y) * w.W + x;
      __stcg(w.cand + (is_wall ? at + __popc(bw & below) : other + __popc(bo & below)), (uint32_t)i);
      __stcg(w.label + i, (uint32_t)i);
      __stcg(r.Wg + i, -__ldcg(r.Wg + i));  // marked
    }
    at += __popc(bw);
    other += __popc(bo);
  }
}

// The whole block: follows what did not fit a front (cells marked kActive).  The
// block looks through its share of the flags; *again = whether any did not fit.
__device__ void wide_rest(const Resolve& r, Front& f, unsigned int& steps) {
  const FillWork& w = r.w;
  const int64_t words = ((int64_t)w.W * w.H + 15) / 16;  // (the flags' space is a multiple of 256)
  const int64_t share = (words + gridDim.x - 1) / gridDim.x;
  const int64_t b0 = share * blockIdx.x, b1 = min(b0 + share, words);
  unsigned int work = 0;
  for (int64_t base = b0; base < b1; base += blockDim.x) {
    __syncthreads();
    if (threadIdx.x < 3) f.n[threadIdx.x] = 0;
    __syncthreads();
    if (base + threadIdx.x < b1) {
      const int64_t c16 = (base + threadIdx.x) * 16;
      const uint4 v = __ldcg(reinterpret_cast<const uint4*>(w.flags + c16));
      const unsigned int f4[4] = {v.x, v.y, v.z, v.w};
      static_assert(kActive == 1, "the low bit of each flag byte");
#pragma unroll
      for (int k = 0; k < 4; k++)
        for (unsigned int m = f4[k] & 0x01010101u; m; m &= m - 1) {
          const int64_t c = c16 + 4 * k + ((__ffs(m) - 1) >> 3);
          r.clear(c, kActive);
          __threadfence();  // a fall after the read below marks the cell again
          // (Of a wall just confirmed: its component's minimum is used up.)
          if (r.get(c) & kUnsureWall) __stcg(w.aux + __ldcg(w.label + c), 0xffffffffu);
          front_push(r, f, 0, 0, (uint32_t)c, r.level(c));
        }
    }
    follow<false, 0>(r, f, 0u, 0u, steps, work);
  }
}

// The phases over the nq walls at the list's start, all levels marked.
// Returns their number.
__device__ int wide_phases(const Resolve& r, Front& f, unsigned int nq, bool* ok) {
  const FillWork& w = r.w;
  const unsigned int nblocks = gridDim.x;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const unsigned int gwarp = blockIdx.x * warps + (threadIdx.x >> 5), nwarps = nblocks * warps;
  unsigned int more = 0, steps = 0, work = 0;
  int phases = 0;
  // A warp's entries: groups of 32 at a stride, so that each warp has a part of
  // every lake.  Those still pending are kept at the front of its own places.
  auto place = [&](unsigned int k) { return ((k >> 5) * nwarps + gwarp) * 32u + (k & 31u); };
  const unsigned int groups = (nq + 31u) / 32u;
  unsigned int len = groups > gwarp ? (groups - gwarp + nwarps - 1) / nwarps * 32u : 0u;
  if (len && place(len - 1) >= nq) len -= place(len - 1) - (nq - 1);
  // fn(c) for each entry; it stays if that is true.
  auto sift = [&](auto fn) {
    unsigned int out = 0;
    for (unsigned int k0 = 0; k0 < len; k0 += 32) {
      const bool in = k0 + lane < len;
      const uint32_t c = in ? __ldcg(w.cand + place(k0 + lane)) : 0u;
      const bool keep = in && fn(c);
      const unsigned int ball = __ballot_sync(0xffffffffu, keep);
      const unsigned int to = out + __popc(ball & ((1u << lane) - 1u));
      if (keep && to != k0 + lane) __stcg(w.cand + place(to), c);
      out += __popc(ball);
    }
    __syncwarp();
    len = out;
  };
  while (*ok) {
    // The least level of each component's pending walls (above their q).
    __syncthreads();
    if (threadIdx.x < 3) f.n[threadIdx.x] = 0;
    if (threadIdx.x == 0) f.full = f.nfresh = 0;
    bool some = false;
    sift([&](uint32_t c) {
      const float lv = r.level(c);
      if (!(lv > r.q[c])) return false;  // for good: levels only fall
      if (lv < kInf) {
        const uint32_t root = __ldcg(w.label + c);
        // Every label is a root: a cell labelled otherwise would take a minimum
        // nothing resets.
        if (phases == 0 && __ldcg(w.label + root) != root) atomicCAS((int*)(w.scal + S_ERR), 0, 6);
        if (__float_as_uint(lv) < __ldcg(w.aux + root)) atomicMin(&w.aux[root], __float_as_uint(lv));
        some = true;
      }
      return true;
    });
    if (!any_of(w, f, nblocks, some, &more, ok)) break;
    // Each phase confirms at least one cell of every component with a pending
    // one (the cell holding its minimum).
    if (++phases > (int)min(nq, 0x7fffff00u) + 8) {
      if (threadIdx.x == 0) atomicCAS((int*)(w.scal + S_ERR), 0, 5);
      break;  // (in every block)
    }
    sift([&](uint32_t c) {
      const unsigned int m = __ldcg(w.aux + __ldcg(w.label + c));
      if (m == 0xffffffffu || !(r.q[c] <= __uint_as_float(m))) return true;
      r.set(c, kConfirmed);
      const float lv = r.level(c);
      if (lv < kInf) front_push(r, f, 0, 0, c, lv);
      return false;
    });
    any_of(w, f, nblocks, false, &more, ok);
    if (!*ok) break;
    // The minima that were used are reset: the cell that holds one is among
    // those just confirmed.
    for (int e = threadIdx.x; e < min(f.n[0], kFrontCells); e += blockDim.x)
      __stcg(w.aux + __ldcg(w.label + f.cell[0][e]), 0xffffffffu);
    follow<false, 0>(r, f, 0u, 0u, steps, work);
    for (;;) {
      __syncthreads();
      const bool full = f.full != 0;
      if (!any_of(w, f, nblocks, full, &more, ok)) break;
      if (threadIdx.x == 0) f.full = 0;
      wide_rest(r, f, steps);
    }
  }
  return phases;
}

template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1)
fill_resolve_wide_kernel(LevelArgs a, Resolve r, int flood_warps) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const FillWork& w = a.w;
  volatile unsigned int* vs = w.scal;
  if (!vs[S_WIDE] || vs[S_ERR]) return;  // (final before the launch)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int gwarp = blockIdx.x * warps + warp, nwarps = gridDim.x * warps;
  const int ntiles = w.tiles_x * w.tiles_y;
  GridSync gs{w.scal + S_BAR_COUNT, w.scal + S_BAR_GEN, (int*)(w.scal + S_ERR)};
  LevelSmem& s = reinterpret_cast<LevelSmem*>(smraw)[warp];
  const unsigned long long t0 = global_ns();
  // A flood from the levels and masks that `start` leaves in every tile.
  auto flood = [&](auto start) -> bool {
    for (int t = gwarp; t < ntiles; t += nwarps) start(t);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      vs[S_HEAD] = 0u;  // (the queue is empty, abandoned tickets aside)
      vs[S_TAIL] = 0u;
      vs[S_DONE] = 0u;
    }
    if (!grid_barrier(gs, gridDim.x)) return false;
    if (!seed_queue(w, gs, gwarp, nwarps, lane, ntiles)) return false;
    if (warp < flood_warps)
      drain(w, lane, ntiles, false, [&](int t, VisitStats& st) {
        level_visit<false>(s, a, fill_queue(w), t, lane, st);
      });
    // (A failure is in the error word.)
    return grid_barrier(gs, gridDim.x) && !__syncthreads_or(vs[S_ERR] != 0u);
  };
  if (!flood([&](int t) { wide_start_lower(a, t, lane); })) return;
  const unsigned long long t1 = global_ns();
  if (!flood([&](int t) { wide_start_upper(a, t, lane); })) return;
  for (int t = gwarp; t < ntiles; t += nwarps) wide_walls(r, t, lane);
  if (!grid_barrier(gs, gridDim.x)) return;
  for (int t = gwarp; t < ntiles; t += nwarps) wide_between(r, t, lane);
  if (!grid_barrier(gs, gridDim.x)) return;
  // (No mask is read from here on: the labels take their space.)
  const unsigned int nq = vs[S_UNSURE];
  int phases = 0;
  if (nq) {
    for (int t = gwarp; t < ntiles; t += nwarps) wide_list(r, t, lane, nq);
    if (!grid_barrier(gs, gridDim.x)) return;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
    const int64_t no = (int64_t)nq + vs[S_BEHIND];
    bool joined = true;
    for (int64_t j = tid; j < 4 * no; j += nthreads) {  // four threads a cell: W, NW, N, NE
      const int d = (int)(j & 3);
      const uint32_t c = __ldcg(w.cand + (j >> 2));
      const int cx = (int)(c % (uint32_t)w.W), cy = (int)(c / (uint32_t)w.W);
      const int nx = cx + (d == 0 ? -1 : d - 2), ny = cy + (d == 0 ? 0 : -1);
      if (nx < 0 || ny < 0 || nx >= w.W) continue;
      const uint32_t n = (uint32_t)ny * (uint32_t)w.W + (uint32_t)nx;
      if (r.get(n) & kUnsure) joined &= uf_unite(w.label, c, n);
    }
    if (!joined) atomicCAS((int*)(w.scal + S_ERR), 0, 6);
    if (!grid_barrier(gs, gridDim.x)) return;
    // From here aux holds the components' least pending level (at their roots).
    for (int64_t j = tid; j < nq; j += nthreads) {
      const uint32_t c = __ldcg(w.cand + j), root = uf_root(w.label, c);
      w.label[c] = root;
      __stcg(w.aux + root, 0xffffffffu);
    }
    if (!grid_barrier(gs, gridDim.x)) return;
    Front& front = *reinterpret_cast<Front*>(smraw);
    if (threadIdx.x == 0) front.gen = vs[S_BAR_GEN];  // (any_of fences before it arrives)
    __syncthreads();
    bool ok = true;
    phases = wide_phases(r, front, nq, &ok);
    if (!ok) return;
  }
  // The marks come off, and cells no outlet reached keep q.
  for (int t = gwarp; t < ntiles; t += nwarps) {
    const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
    for (int y = y0; y < min(y0 + kTile, w.H) && x < w.W; y++) {
      const int64_t i = (int64_t)y * w.W + x;
      const float qv = r.q[i], v = __ldcg(r.Wg + i), lv = fabsf(v);
      if (qv == r.nodata) continue;
      const float n = lv == kInf ? qv : lv;
      if (__float_as_uint(n) != __float_as_uint(v)) r.Wg[i] = n;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const unsigned long long t2 = global_ns();
    vs[S_PASS] = vs[S_PASS] + 4u + (unsigned int)phases;
    vs[S_PHASES] = (unsigned int)phases;
    vs[S_US_B] = vs[S_US_B] + (unsigned int)((t1 - t0) / 1000);
    vs[S_US_P] = (unsigned int)((t2 - t1) / 1000);
  }
}

__global__ void quantize_min_kernel(float* __restrict__ d, int W, int H, float nodata,
                                    unsigned int* minslot, uint8_t* __restrict__ tseed,
                                    int tiles_x) {
  const unsigned int i = blockIdx.x * blockDim.x + threadIdx.x;
  float m = kInf;
  if (i < (unsigned int)W * (unsigned int)H) {
    const float q = fill_quantize(d[i], nodata);
    d[i] = q;
    m = q;
    const int y = (int)(i / (unsigned int)W), x = (int)(i - (unsigned int)y * (unsigned int)W);
    if (q == 0.0f || x == 0 || y == 0 || x == W - 1 || y == H - 1)
      tseed[(y / kTile) * tiles_x + x / kTile] = 1;
  }
  unsigned int o = float_to_ordered(m);
  o = __reduce_min_sync(0xffffffffu, o);
  // One atomic per block (same-address atomics from every warp queue up).
  __shared__ unsigned int bmin;
  if (threadIdx.x == 0) bmin = 0xffffffffu;
  __syncthreads();
  if ((threadIdx.x & 31) == 0) atomicMin(&bmin, o);
  __syncthreads();
  if (threadIdx.x == 0) atomicMin(minslot, bmin);
}

// Blocks and warps per block of a flood over `ntiles` tiles: one block on
// every SM (`blocks` of them) as far as there are tiles, with as many warps
// as the tiles can keep busy.  At 512^2 (256 tiles) a visit takes half as
// long with 2 warps on each of 128 SMs as with 20 warps on each of 13.
static void flood_shape(int ntiles, int blocks, int warps, int* grid, int* per_block) {
  *grid = std::max(1, std::min(blocks, ntiles));
  *per_block = std::max(1, std::min(warps, (ntiles + *grid - 1) / *grid));
}

template <bool MARKS, int WARPS>
static cageo_status launch_level_warps(const LevelArgs& a, cudaStream_t s) {
  const size_t smem = sizeof(LevelSmem) * WARPS;
  auto fn = level_flood_kernel<MARKS, WARPS>;
  static PerDevice resident;  // one table per instantiation
  int blocks = 0;
  cageo_status st = per_device(resident, &blocks, [&](int dev, int* v) -> cageo_status {
    CAGEO_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return resident_blocks((const void*)fn, WARPS * 32, smem, dev, v);
  });
  if (st) return st;
  int grid, per;
  flood_shape(a.w.tiles_x * a.w.tiles_y, blocks, WARPS, &grid, &per);
  LevelArgs args = a;
  void* params[] = {&args};
  CAGEO_CUDA(cudaLaunchCooperativeKernel((const void*)fn, dim3(grid), dim3(per * 32), params,
                                         sizeof(LevelSmem) * per, s));
  return CAGEO_OK;
}

bool fill_flood_warps_valid(int warps) { return warps == 16 || warps == 20 || warps == 22; }

template <bool MARKS>
static cageo_status launch_level(const LevelArgs& a, cudaStream_t s) {
  switch (a.w.flood_warps) {
    case 16: return launch_level_warps<MARKS, 16>(a, s);
    case 20: return launch_level_warps<MARKS, 20>(a, s);
    case 22: return launch_level_warps<MARKS, 22>(a, s);
  }
  set_error("pit filling: %d warps per block is not one of 16, 20, 22", a.w.flood_warps);
  return CAGEO_ERR_ARGUMENT;
}

static cageo_status launch_resolve(const Resolve& r, cudaStream_t s) {
  static PerDevice resident;
  int blocks = 0;
  cageo_status st = per_device(resident, &blocks, [&](int dev, int* v) -> cageo_status {
    return resident_blocks((const void*)fill_resolve_kernel, kResolveThreads, 0, dev, v);
  });
  if (st) return st;
  Resolve args = r;
  void* params[] = {&args};
  // Blocks for lists of up to 1 cell in 128 (walls above their q are 1 in 600 on
  // terrain; blocks take several turns on longer lists).  All of them have to
  // find room on the GPU at once, beside what other streams run.
  const int64_t n = (int64_t)r.w.W * r.w.H;
  const int grid = (int)std::min<int64_t>(blocks, (n + 128 * kResolveShare - 1) / (128 * kResolveShare));
  CAGEO_CUDA(cudaLaunchCooperativeKernel((const void*)fill_resolve_kernel, dim3(grid),
                                         dim3(kResolveThreads), params, 0, s));
  return CAGEO_OK;
}

// The wide resolution: a block per SM, of which a small grid's floods use as many
// warps as the flood would.
static cageo_status launch_resolve_wide(const LevelArgs& a, const Resolve& r, cudaStream_t s) {
  constexpr int kWarps = 20;
  constexpr size_t kSmem = sizeof(LevelSmem) * kWarps;
  static_assert(kSmem >= sizeof(Front), "the front lies in the tiles' space");
  auto fn = fill_resolve_wide_kernel<kWarps>;
  static PerDevice resident;
  int blocks = 0;
  cageo_status st = per_device(resident, &blocks, [&](int dev, int* v) -> cageo_status {
    CAGEO_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    return resident_blocks((const void*)fn, kWarps * 32, kSmem, dev, v);
  });
  if (st) return st;
  int grid, per;
  flood_shape(a.w.tiles_x * a.w.tiles_y, blocks, kWarps, &grid, &per);
  LevelArgs la = a;
  Resolve lr = r;
  void* params[] = {&la, &lr, &per};
  CAGEO_CUDA(cudaLaunchCooperativeKernel((const void*)fn, dim3(grid), dim3(kWarps * 32), params,
                                         kSmem, s));
  return CAGEO_OK;
}

cageo_status fill_begin(const FillWork& w, cudaStream_t s) {
  const int ntiles = w.tiles_x * w.tiles_y;
  // 8 rim words (16 bytes each) per thread, but no more blocks than fill the GPU.
  const unsigned blocks = (unsigned)std::min<int64_t>(
      2048, ((int64_t)ntiles * (kRimCells / 2) + kRingSlack + 1023) / 1024);
  fill_begin_kernel<<<blocks, 256, 0, s>>>(w, ntiles);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

static unsigned warp_per_tile_blocks(size_t nt) { return (unsigned)((nt + 7) / 8); }

static LevelArgs walled_args(const float* q, float* filled, const FillWork& w, float nodata) {
  return LevelArgs{q, filled, w, nodata, w.slab_min ? w.slab_min : w.scal + S_MIN, 0, 0};
}

static Resolve resolve_args(const LevelArgs& a) {
  return Resolve{a.q, a.Wg, a.w, a.nodata, a.minslot, a.w.slab_h ? a.w.slab_h : a.w.H};
}

cageo_status fill_run(const float* q, float* filled, const FillWork& w, float nodata,
                      cudaStream_t s) {
  const unsigned tblocks = warp_per_tile_blocks((size_t)w.tiles_x * w.tiles_y);
  if (!w.seeded) fill_seed_kernel<<<tblocks, 256, 0, s>>>(q, w);
  const LevelArgs a = walled_args(q, filled, w, nodata);
  if (w.marks) CAGEO_CUDA(cudaEventRecord(w.marks[0], s));
  cageo_status st = launch_level<false>(a, s);
  if (st) return st;
  if (w.marks) CAGEO_CUDA(cudaEventRecord(w.marks[1], s));
  fill_walls_kernel<<<tblocks, 256, 0, s>>>(a);
  CAGEO_CUDA(cudaGetLastError());
  if (w.marks) CAGEO_CUDA(cudaEventRecord(w.marks[2], s));
  const Resolve r = resolve_args(a);
  if ((st = launch_resolve(r, s))) return st;
  if (w.wide && (st = launch_resolve_wide(a, r, s))) return st;
  if (w.marks) CAGEO_CUDA(cudaEventRecord(w.marks[3], s));
  return CAGEO_OK;
}

cageo_status fill_run_exact(const float* v, float* filled, const FillWork& w, float nodata,
                            const float* warm, cudaStream_t s) {
  const int64_t n = (int64_t)w.W * w.H;
  const size_t nt = (size_t)w.tiles_x * w.tiles_y;
  const unsigned tblocks = warp_per_tile_blocks(nt);
  LevelArgs a{v, filled, w, nodata, nullptr, warm ? 1 : 0, 0};
  if (!warm) {
    if (!w.seeded) fill_seed_kernel<<<tblocks, 256, 0, s>>>(v, w);
    cageo_status st = launch_level<false>(a, s);
    if (st) return st;
  } else {
    // A warm start may hold values above the answer anywhere: every tile is
    // visited.  After the warm flood with support marks, the unsupported
    // cells restart from +inf and the repair flood visits their tiles.
    CAGEO_CUDA(cudaMemsetAsync(w.tseed, 1, nt, s));
    fill_warm_start_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(v, warm, filled, n);
    cageo_status st = launch_level<true>(a, s);
    if (st) return st;
    fill_unsupported_kernel<<<tblocks, 256, 0, s>>>(a);
    CAGEO_CUDA(cudaGetLastError());
    a.stage = 3;
    a.warm = 0;
    if ((st = launch_level<false>(a, s))) return st;
  }
  fill_final_exact_kernel<<<tblocks, 256, 0, s>>>(a);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

cageo_status fill_quantize_min(float* d, const FillWork& w, float nodata, cudaStream_t s) {
  const int64_t n = (int64_t)w.W * w.H;
  quantize_min_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
      d, w.W, w.H, nodata, w.scal + S_MIN, w.tseed, w.tiles_x);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

// Adds a warm-started exact fill's counters to acc (device, 9 entries):
// fills, fills that restarted any cell, cells restarted, tile visits and
// sweep rounds of the warm flood, sweep rounds of the repair flood,
// microseconds of the warm and of the repair flood, repair tile visits.
__global__ void fill_warm_stats_kernel(const unsigned int* __restrict__ scal,
                                       unsigned long long* acc) {
  if (threadIdx.x != 0) return;
  const unsigned int reset = scal[S_RESET];
  acc[0] += 1;
  acc[1] += reset ? 1 : 0;
  acc[2] += reset;
  acc[3] += scal[S_TILES_A];
  acc[4] += scal[S_ROUNDS_A];
  acc[5] += scal[S_ROUNDS_B];
  acc[6] += scal[S_US_A];
  acc[7] += scal[S_US_B];
  acc[8] += scal[S_TILES_B];
}

cageo_status fill_accumulate_warm_stats(const FillWork& w, unsigned long long* acc,
                                        cudaStream_t s) {
  fill_warm_stats_kernel<<<1, 32, 0, s>>>(w.scal, acc);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

const unsigned int* fill_error_word(const FillWork& w) { return w.scal + S_ERR; }

const char* fill_error_text(unsigned int error) {
  static const char* what[] = {"",
                               "a grid-wide wait hit its limit",
                               "a warp waited for a tile past its limit",
                               "a tile's queue state kept changing",
                               "the tile visits or relaxation rounds passed their limit",
                               "the confirmation phases passed their limit",
                               "the labels of the unsettled cells are not settled roots"};
  return error < 7 ? what[error] : "unknown error";
}

const unsigned int* fill_wide_word(const FillWork& w) { return w.scal + S_WIDE; }

static cageo_status check_scalars(const unsigned int (&h)[S_SIZE], int64_t* stats) {
  if (stats) {
    stats[0] = h[S_PASS];
    stats[1] = h[S_PHASES];
    stats[2] = h[S_PASSES_A];
    stats[3] = h[S_STEPS];
    stats[4] = h[S_US_A];
    stats[5] = h[S_US_B];
    stats[6] = h[S_US_P];
    stats[7] = h[S_TILES_A];
    stats[8] = h[S_ROUNDS_A];
    stats[9] = h[S_TILES_B] ? h[S_TILES_B] : h[S_CAND] + h[S_MORE];
    stats[10] = h[S_ROUNDS_B];
    stats[11] = h[S_KCYC_LOAD];
    stats[12] = h[S_KCYC_SWEEP];
    stats[13] = h[S_KCYC_STORE];
    stats[14] = h[S_KCYC_IDLE_A];
    stats[15] = h[S_KCYC_IDLE_B];
    stats[16] = h[S_RESET];
  }
  if (h[S_ERR]) {
    set_error("pit filling: %s (tiles finished %u, phases %u, listed cells %u)",
              fill_error_text(h[S_ERR]), h[S_DONE], h[S_PHASES], h[S_CAND]);
    return CAGEO_ERR_NO_CONVERGENCE;
  }
  return CAGEO_OK;
}

cageo_status fill_check_status(const FillWork& w, int64_t* stats) {
  unsigned int h[S_SIZE];
  CAGEO_CUDA(cudaMemcpy(h, w.scal, sizeof(h), cudaMemcpyDeviceToHost));
  return check_scalars(h, stats);
}

cageo_status fill_finish(const float* q, float* filled, const FillWork& w, float nodata,
                         int64_t* stats, cudaStream_t s) {
  unsigned int h[S_SIZE];
  CAGEO_CUDA(cudaStreamSynchronize(s));
  CAGEO_CUDA(cudaMemcpy(h, w.scal, sizeof(h), cudaMemcpyDeviceToHost));
  if (h[S_WIDE] && !h[S_ERR]) {
    const LevelArgs a = walled_args(q, filled, w, nodata);
    const cageo_status st = launch_resolve_wide(a, resolve_args(a), s);
    if (st) return st;
    CAGEO_CUDA(cudaStreamSynchronize(s));
    CAGEO_CUDA(cudaMemcpy(h, w.scal, sizeof(h), cudaMemcpyDeviceToHost));
  }
  return check_scalars(h, stats);
}

}  // namespace cageo

using namespace cageo;

extern "C" cageo_status cageo_pitfill_exact_warm(const float* d_dem, const float* d_warm,
                                                 float* d_filled, int W, int H, float nodata_dem,
                                                 void* d_workspace, size_t workspace_bytes,
                                                 int64_t* h_stats, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_dem && d_filled && valid_dims(W, H), "pointers and size");
  CAGEO_CHECK_ARG(W <= 65535 && H <= 65535, "width and height must be <= 65535");
  CAGEO_CHECK_ARG(d_dem != d_filled && d_warm != d_filled, "the filled grid must not alias");
  Scratch ws;
  cageo_status st = ws.acquire(d_workspace, workspace_bytes, fill_workspace_bytes(W, H), stream);
  if (st) return st;
  FillWork w = fill_carve(ws.ptr, W, H);
  if ((st = fill_begin(w, stream))) return st;
  if ((st = fill_run_exact(d_dem, d_filled, w, nodata_dem, d_warm, stream))) return st;
  CAGEO_CUDA(cudaStreamSynchronize(stream));
  return fill_check_status(w, h_stats);
}

extern "C" size_t cageo_pitfill_workspace_size(int W, int H) {
  if (!valid_dims(W, H)) return 0;
  return fill_workspace_bytes(W, H);
}

extern "C" cageo_status cageo_pitfill(float* d_dem, float* d_filled, int W, int H,
                                      float nodata_dem, int mode, void* d_workspace,
                                      size_t workspace_bytes, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_dem && d_filled && valid_dims(W, H), "pointers and size");
  CAGEO_CHECK_ARG(W <= 65535 && H <= 65535, "width and height must be <= 65535");
  CAGEO_CHECK_ARG(d_dem != d_filled, "the filled grid must not alias the DEM");
  CAGEO_CHECK_ARG(mode == CAGEO_FILL_CPU_COMPAT || mode == CAGEO_FILL_EXACT, "fill mode");
  Scratch ws;
  cageo_status st = ws.acquire(d_workspace, workspace_bytes, fill_workspace_bytes(W, H), stream);
  if (st) return st;
  FillWork w = fill_carve(ws.ptr, W, H);
  if ((st = fill_begin(w, stream))) return st;
  if (mode == CAGEO_FILL_EXACT) {
    if ((st = fill_run_exact(d_dem, d_filled, w, nodata_dem, nullptr, stream))) return st;
  } else {
    if ((st = fill_quantize_min(d_dem, w, nodata_dem, stream))) return st;
    w.seeded = true;
    if ((st = fill_run(d_dem, d_filled, w, nodata_dem, stream))) return st;
    return fill_finish(d_dem, d_filled, w, nodata_dem, nullptr, stream);
  }
  CAGEO_CUDA(cudaStreamSynchronize(stream));
  return fill_check_status(w, nullptr);
}
