// trace_border.cu -- A8 flow tracing by pointer jumping and A9 catchment
// border extraction + Monte Carlo accumulation.
//
// Tracing (src/flowtracing/FlowTracingAlgorithmCPUOpenMP.h:34-134): a stream
// cell (streams >= 0) is LAKE; every other cell follows its direction until
// it leaves the grid (OUTSIDE) or steps onto a stream cell s (label
// (int)(-streams[s])).  The reference walks each path serially with caching;
// the label of a cell depends only on where its path ends, so here every
// cell holds a packed 32-bit state -- "points to cell p" or "resolved to
// label l".  Paths are first followed inside each 32x32 tile; a path that
// leaves its tile then points at the border cell of the next tile it
// enters, and those border cells (124 per tile, kept in a compact array)
// point only at border cells of other tiles.  Pointer doubling
// (p <- state[p]) over the compact array resolves them in O(log path
// length) passes over 12% of the cells; every other cell then needs one
// lookup.  A cell without a direction
// (0,0) is a dead end: the reference's walk never terminates there, leaves
// the path at 0 and its connect pass then copies the label of cell 0; such
// cells and label-0 terminals take the label of cell 0 here too (or, in the
// dead-end-error mode used with the GPU path's semantics, dead ends and the
// cells draining into them are ERROR).  (The
// reference also abandons walks longer than 100000 steps; paths of that
// length do not occur in these grids and are not modelled.)
//
// Border (src/catchmentborder/CatchmentBorderAlgorithmCPUOpenMP.h:30-82):
// border = 1 where the label is not LAKE and some N8 neighbour has a larger
// label that is not LAKE; the count grid adds it
// (src/catchmentborder/CatchmentBorderAlgorithm.h:53-74).
#include <algorithm>
#include "common.cuh"
#include "front.cuh"
#include "routing.cuh"
#include "stage_math.cuh"

namespace cageo {

// Packed per-cell state (int32): >= 0 points to a cell; < 0 is resolved,
// holding code(label) = label - 1 (labels are <= 0, so label 0 stays
// negative); kStuckCode marks a dead end.  Stream values whose negation
// does not fit (|streams| >= 2^31 - 1) are outside the supported range.
constexpr int kStuckCode = (int)0x80000000;
constexpr int kJumpThreads = 256;
enum : int { T_ERR = 2, T_ACTIVE = 3, T_JUMPS = 6, T_BAR_COUNT = kBarCountSlot,
             T_BAR_GEN = kBarGenSlot, T_SIZE = kScalarSlots };

__device__ __forceinline__ int label_code(int label) { return label - 1; }

constexpr int kBorderCells = 124;  // cells on the rim of a 32x32 tile

size_t trace_workspace_bytes(int W, int H) {
  const size_t n = (size_t)W * H;
  const size_t nt = (size_t)((W + 31) / 32) * ((H + 31) / 32);
  return align_up(n * 4, 256) + align_up(nt * kBorderCells * 4, 256) + 512;
}

TraceWork trace_carve(void* base, int W, int H) {
  TraceWork w;
  w.W = W;
  w.H = H;
  w.tiles_x = (W + 31) / 32;
  w.tiles_y = (H + 31) / 32;
  const size_t n = (size_t)W * H;
  const size_t nt = (size_t)w.tiles_x * w.tiles_y;
  char* p = (char*)base;
  w.state = (int*)p;
  p += align_up(n * 4, 256);
  w.bstate = (int*)p;
  p += align_up(nt * kBorderCells * 4, 256);
  w.scal = (unsigned int*)p;
  return w;
}

// Compact index of cell (x, y) on the rim of its 32x32 tile (x % 32 or
// y % 32 is 0 or 31): top row 0..31, bottom row 32..63, left column rows
// 1..30 at 64..93, right column rows 1..30 at 94..123.
__device__ __forceinline__ int border_index(int x, int y, int tiles_x) {
  const int lx = x & 31, ly = y & 31;
  const int b = ly == 0 ? lx : ly == 31 ? 32 + lx : lx == 0 ? 63 + ly : 93 + ly;
  return ((y >> 5) * tiles_x + (x >> 5)) * kBorderCells + b;
}

// While paths are followed inside a tile, a state from here on points at one of
// the tile's 1024 cells (rim indices stay below it).
constexpr int kInTile = 0x7ffffc00;

// Initial state of every cell, then pointer jumping inside its 32x32 tile in
// shared memory: each cell ends resolved (a label or a dead end) or pointing
// at the first cell of its path outside the tile, so the global jumps hop from
// tile to tile.  One block per tile, 4 cells of a row per thread.  The jumps
// need no barriers: a cell's word only ever moves on along its own path, so
// whichever version a thread reads is right, and a newer one is nearer the
// end.  Bound by instruction issue and the shared-memory chase: 0.34 ms at
// 8192^2 where a cell per thread and two barriers a round took 0.48.
// CODE: whether a cell is a stream comes from the burn codes (1 byte; streams
// is read only where a path ends), otherwise from the streams themselves.
template <bool CODE>
__global__ void __launch_bounds__(256) trace_init_kernel(const char2* __restrict__ dir,
                                                         const float* __restrict__ streams,
                                                         const uint8_t* __restrict__ code,
                                                         TraceWork w, int aligned) {
  __shared__ __align__(16) int cell[32 * 32];
  __shared__ unsigned int smask[32];  // stream cells of the tile's rows
  const int W = w.W, H = w.H, slab_h = w.slab_h ? w.slab_h : H;
  const int ly = threadIdx.x >> 3, lx = (threadIdx.x & 7) * 4;
  const int x = blockIdx.x * 32 + lx, y = blockIdx.y * 32 + ly;
  const int slab = y / slab_h, ys = y - slab * slab_h;
  const int64_t i = (int64_t)y * W + x, is = (int64_t)ys * W + x;
  const bool in = y < H && x < W;
  char2 d[4];
  unsigned int sbits = 0;
  if (aligned && in) {  // W is a multiple of 4: all four cells or none
    const uint2 v = *reinterpret_cast<const uint2*>(dir + i);
    d[0] = make_char2((signed char)v.x, (signed char)(v.x >> 8));
    d[1] = make_char2((signed char)(v.x >> 16), (signed char)(v.x >> 24));
    d[2] = make_char2((signed char)v.y, (signed char)(v.y >> 8));
    d[3] = make_char2((signed char)(v.y >> 16), (signed char)(v.y >> 24));
    if (CODE) {
      const unsigned int c = *reinterpret_cast<const unsigned int*>(code + is);
      static_assert(kCodeTraceStream == 0x40, "bit 6 of a code");
      sbits = (c >> 6 & 1u) | (c >> 14 & 1u) << 1 | (c >> 22 & 1u) << 2 | (c >> 30 & 1u) << 3;
    } else {
      const float4 f = *reinterpret_cast<const float4*>(streams + is);
      sbits = (f.x >= 0.0f ? 1u : 0u) | (f.y >= 0.0f ? 2u : 0u) | (f.z >= 0.0f ? 4u : 0u) |
              (f.w >= 0.0f ? 8u : 0u);
    }
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      d[k] = make_char2(0, 0);
      if (!in || x + k >= W) continue;
      d[k] = dir[i + k];
      if (CODE ? (code[is + k] & kCodeTraceStream) != 0 : streams[is + k] >= 0.0f) sbits |= 1u << k;
    }
  }
  unsigned int m = sbits << lx;  // the row's mask: 8 threads of a warp hold a row
  m |= __shfl_xor_sync(0xffffffffu, m, 1);
  m |= __shfl_xor_sync(0xffffffffu, m, 2);
  m |= __shfl_xor_sync(0xffffffffu, m, 4);
  if ((threadIdx.x & 7) == 0) smask[ly] = m;
  __syncthreads();
  int s[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    s[k] = kStuckCode;
    if (!in || x + k >= W) continue;
    const int nx = x + k + d[k].x, nys = ys + d[k].y;
    if (sbits >> k & 1u) {
      s[k] = label_code(kLake);
    } else if (nx < 0 || nx >= W || nys < 0 || nys >= slab_h) {
      s[k] = label_code(kOutside);
    } else if (d[k].x != 0 || d[k].y != 0) {
      const int tx = lx + k + d[k].x, ty = ly + d[k].y;
      const bool inside = tx >= 0 && tx < 32 && ty >= 0 && ty < 32;
      const int64_t n = (int64_t)nys * W + nx;
      bool stream;
      if (inside) stream = smask[ty] >> tx & 1u;
      else stream = CODE ? (code[n] & kCodeTraceStream) != 0 : streams[n] >= 0.0f;
      if (stream) s[k] = label_code((int)(-streams[n]));
      else if (inside) s[k] = kInTile | (ty * 32 + tx);
      else s[k] = border_index(nx, y + d[k].y, w.tiles_x);  // on the rim of the next tile
    }
  }
  volatile int* c = cell;
  const int li = ly * 32 + lx;
  *reinterpret_cast<int4*>(&cell[li]) = make_int4(s[0], s[1], s[2], s[3]);
  __syncthreads();
  auto in_tile = [](int v) { return v >= kInTile; };
  // A path of a 32x32 tile has at most 1024 cells: one still inside after as
  // many steps is on a cycle, which never resolves (reported as an error).
  bool any = true;
  for (int it = 0; any && it < 1056; it++) {
    any = false;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (in_tile(s[k])) {
        s[k] = c[s[k] & 1023];
        c[li + k] = s[k];
        any |= in_tile(s[k]);
      }
    }
  }
  if (any) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (in_tile(s[k])) s[k] = kStuckCode;
    atomicCAS((int*)(w.scal + T_ERR), 0, 2);
  }
  // (The state array is workspace: aligned where W is a multiple of 4.)
  if (!in) {
  } else if ((W & 3) == 0) {
    *reinterpret_cast<int4*>(w.state + i) = make_int4(s[0], s[1], s[2], s[3]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (x + k < W) w.state[i + k] = s[k];
  }
  // The whole rim is written: the jumps run over entries outside the grid too.
  int* b = w.bstate + ((int64_t)blockIdx.y * w.tiles_x + blockIdx.x) * kBorderCells;
  if (ly == 0) *reinterpret_cast<int4*>(b + lx) = make_int4(s[0], s[1], s[2], s[3]);
  else if (ly == 31) *reinterpret_cast<int4*>(b + 32 + lx) = make_int4(s[0], s[1], s[2], s[3]);
  else if (lx == 0) b[63 + ly] = s[0];
  else if (lx == 28) b[93 + ly] = s[3];
}

// Pointer doubling in place over the tiles' border cells (reading a
// neighbour's newer state only speeds convergence).  Each thread takes 4 cells
// per iteration so their dependent load pairs overlap.  Persistent; one bounded
// grid barrier per pass.
__global__ void __launch_bounds__(kJumpThreads, 8) trace_jump_kernel(int* st, TraceWork w) {
  const int64_t N = (int64_t)w.tiles_x * w.tiles_y * kBorderCells;
  GridSync gs{w.scal + T_BAR_COUNT, w.scal + T_BAR_GEN, (int*)(w.scal + T_ERR)};
  volatile unsigned int* vs = w.scal;
  const int64_t nthreads = (int64_t)gridDim.x * blockDim.x;
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int pass = 0;
  while (true) {
    // Slot pass%3 is written during this pass and read after its barrier;
    // slot (pass+1)%3 was last read before the previous barrier.
    if (blockIdx.x == 0 && threadIdx.x == 0) vs[T_ACTIVE + (pass + 1) % 3] = 0u;
    bool active = false;
    for (int64_t base = tid; base < N; base += 4 * nthreads) {
      int s[4], t[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int64_t i = base + k * nthreads;
        s[k] = i < N ? st[i] : -1;
      }
#pragma unroll
      for (int k = 0; k < 4; k++) t[k] = s[k] >= 0 ? ((volatile int*)st)[s[k]] : s[k];
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if (s[k] >= 0) {
          st[base + k * nthreads] = t[k];
          active |= t[k] >= 0;
        }
      }
    }
    // One flag update per block: same-address atomics from every warp would
    // queue up at the memory system.
    if (__syncthreads_or(active) && threadIdx.x == 0) atomicOr(&w.scal[T_ACTIVE + pass % 3], 1u);
    if (!grid_barrier(gs, gridDim.x)) break;
    if (vs[T_ACTIVE + pass % 3] == 0u) break;
    if (++pass > 64) {  // 2^64 exceeds any path length: a cycle
      if (threadIdx.x == 0) atomicCAS((int*)(w.scal + T_ERR), 0, 2);
      break;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) vs[T_JUMPS] = (unsigned int)(pass + 1);
}

// Resolved state of a cell from its own state: a path that left the cell's
// tile takes the (resolved) state of the border cell it entered next.
__device__ __forceinline__ int resolve(int c, const int* __restrict__ bst) {
  return c >= 0 ? bst[c] : c;
}

// Label of a resolved state c: label-0 terminals take the label of cell 0 of
// the grid, and so do dead ends (stuck = 0) unless they are reported as ERROR
// (stuck = kError).  first: the state of cell 0 (of the cell's slab).
__device__ __forceinline__ int decode_label(int c, const int* __restrict__ first,
                                            const int* __restrict__ bst, int stuck) {
  const int l = c == kStuckCode ? stuck : c + 1;
  if (l < 0) return l;
  const int c0 = resolve(*first, bst);
  const int l0 = c0 == kStuckCode ? stuck : c0 + 1;
  return l0 >= 0 ? 0 : l0;
}

__global__ void trace_final_kernel(const int* __restrict__ st, const int* __restrict__ bst,
                                   int* __restrict__ label, int64_t n, int stuck) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  label[i] = decode_label(resolve(st[i], bst), st, bst, stuck);
}

__global__ void trace_scalars_kernel(unsigned int* s) {
  for (int i = threadIdx.x; i < T_SIZE; i += blockDim.x) s[i] = 0u;
}

cageo_status trace_run(const int8_t* dir, const float* streams, const uint8_t* code, int* label,
                       const TraceWork& w, cudaStream_t s, int mode, bool write_labels) {
  const int64_t n = (int64_t)w.W * w.H;
  const unsigned blocks = (unsigned)((n + 255) / 256);
  trace_scalars_kernel<<<1, 128, 0, s>>>(w.scal);
  const dim3 g(w.tiles_x, w.tiles_y);
  // Four cells at once where rows start on 4-cell boundaries.
  const bool rows = (w.W & 3) == 0 && ((uintptr_t)dir & 7u) == 0;
  if (code)
    trace_init_kernel<true><<<g, 256, 0, s>>>((const char2*)dir, streams, code, w,
                                              rows && ((uintptr_t)code & 3u) == 0);
  else
    trace_init_kernel<false><<<g, 256, 0, s>>>((const char2*)dir, streams, code, w,
                                               rows && ((uintptr_t)streams & 15u) == 0);
  CAGEO_CUDA(cudaGetLastError());
  static PerDevice resident;
  int coop = 0;
  cageo_status st = per_device(resident, &coop, [&](int dev, int* v) -> cageo_status {
    return resident_blocks((const void*)trace_jump_kernel, kJumpThreads, 0, dev, v);
  });
  if (st) return st;
  int* stp = w.bstate;
  TraceWork wc = w;
  void* params[] = {(void*)&stp, (void*)&wc};
  // Each thread takes 4 border cells per iteration: no more blocks than
  // that covers.
  const int64_t nb = (int64_t)w.tiles_x * w.tiles_y * kBorderCells;
  const int64_t need = (nb + 4 * kJumpThreads - 1) / (4 * kJumpThreads);
  const int jgrid = (int)std::max<int64_t>(1, std::min<int64_t>(coop, need));
  CAGEO_CUDA(cudaLaunchCooperativeKernel((const void*)trace_jump_kernel, dim3(jgrid),
                                         dim3(kJumpThreads), params, 0, s));
  if (write_labels)
    trace_final_kernel<<<blocks, 256, 0, s>>>(w.state, w.bstate, label, n,
                                              mode == CAGEO_TRACE_DEAD_END_ERROR ? kError : 0);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

const unsigned int* trace_error_word(const TraceWork& w) { return w.scal + T_ERR; }

const char* trace_error_text() { return "pointer jumping hit a wait or pass limit"; }

cageo_status trace_check_status(const TraceWork& w, int64_t* jumps) {
  unsigned int h[T_SIZE];
  CAGEO_CUDA(cudaMemcpy(h, w.scal, sizeof(h), cudaMemcpyDeviceToHost));
  if (jumps) *jumps = h[T_JUMPS];
  if (h[T_ERR]) {
    set_error("flow tracing: %s", trace_error_text());
    return CAGEO_ERR_NO_CONVERGENCE;
  }
  return CAGEO_OK;
}

// ---- A9 -------------------------------------------------------------------
// Staged labels of a 32x32 tile and a one-cell halo, rows of 40 with the
// tile's columns from 4 on (16-byte aligned).  LAKE, which neither is nor makes
// a border, and cells outside the grid are staged as the least integer, so a
// cell is a border exactly when the largest of the 3x3 cells around it
// exceeds its own.  The labels below LAKE move up by one into the place it
// leaves, so that the least integer, a label like any other, stays apart.
constexpr int kBS = 40;
constexpr int kNoLabel = (int)0x80000000;
__device__ __forceinline__ int border_key(int label) {
  return label == kLake ? kNoLabel : label + (label < kLake ? 1 : 0);
}

// Position around the tile of halo cell h (0..131): top and bottom rows with
// the corners, then the sides.
__device__ __forceinline__ void halo_cell(int h, int& x, int& y) {
  if (h < 68) {
    y = h < 34 ? -1 : 32;
    x = (h < 34 ? h : h - 34) - 1;
  } else {
    x = h < 100 ? -1 : 32;
    y = h < 100 ? h - 68 : h - 100;
  }
}

// Border mask (bits 0..3) of the 4 cells from (lx, ly) of the tile; up and
// down say whether the rows above and below belong to the same grid.  The
// maxima of three along the rows are shared by the cells.
__device__ __forceinline__ unsigned int border_of_4(const int* L, int lx, int ly, bool up, bool down) {
  int m[4] = {kNoLabel, kNoLabel, kNoLabel, kNoLabel}, own[4];
#pragma unroll
  for (int r = 0; r < 3; r++) {
    const int* row = L + (ly + r) * kBS + 4 + lx;
    const int4 v = *reinterpret_cast<const int4*>(row);
    if (r == 1) {
      own[0] = v.x; own[1] = v.y; own[2] = v.z; own[3] = v.w;
    }
    if ((r == 0 && !up) || (r == 2 && !down)) continue;
    const int a = row[-1], b = row[4];
    m[0] = max(m[0], max(max(a, v.x), v.y));
    m[1] = max(m[1], max(max(v.x, v.y), v.z));
    m[2] = max(m[2], max(max(v.y, v.z), v.w));
    m[3] = max(m[3], max(max(v.z, v.w), b));
  }
  unsigned int out = 0;
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (own[k] != kNoLabel && m[k] > own[k]) out |= 1u << k;
  return out;
}

// Counts of a label grid: one 32x32 tile per block, 4 cells of a row per
// thread.
template <typename T>
__global__ void __launch_bounds__(256) border_kernel(const int* __restrict__ label,
                                                     T* __restrict__ count, int W, int H) {
  __shared__ __align__(16) int L[34 * kBS];
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
  auto at = [&](int x, int y) {
    return x >= 0 && x < W && y >= 0 && y < H ? border_key(label[(int64_t)y * W + x]) : kNoLabel;
  };
  for (int k = threadIdx.x; k < 32 * 32; k += 256)
    L[((k >> 5) + 1) * kBS + 4 + (k & 31)] = at(x0 + (k & 31), y0 + (k >> 5));
  if (threadIdx.x < 132) {
    int hx, hy;
    halo_cell(threadIdx.x, hx, hy);
    L[(hy + 1) * kBS + 4 + hx] = at(x0 + hx, y0 + hy);
  }
  __syncthreads();
  const int ly = threadIdx.x >> 3, lx = (threadIdx.x & 7) * 4;
  const int x = x0 + lx, y = y0 + ly;
  if (y >= H) return;
  const unsigned int b = border_of_4(L, lx, ly, true, true);
#pragma unroll
  for (int k = 0; k < 4; k++)
    if ((b >> k & 1u) && x + k < W) {
      const int64_t i = (int64_t)y * W + x + k;
      count[i] = count[i] + (T)1;
    }
}

// The same from the resolved trace states: decodes the labels of the tile
// (its cells' paths end at rim cells of other tiles, whose states are
// resolved) and of the halo, which is rim cells itself.  A stack of
// realizations adds its slabs' masks to one count grid, but for a slab whose
// gate is set.  The labels are written
// for realization *last only (the one a caller can still ask for; slab 0 is
// realization *real); last null: for every one.  Bound by the label decode's
// dependent loads: 0.19 ms at 8192^2 (0.29 with a cell per thread, 9 label
// reads a cell and all labels written).
__global__ void __launch_bounds__(256) border_state_kernel(TraceWork w, int* __restrict__ label,
                                                           uint32_t* __restrict__ count,
                                                           const int* __restrict__ gate, int stuck,
                                                           const uint32_t* __restrict__ real,
                                                           const uint32_t* __restrict__ last) {
  __shared__ __align__(16) int L[34 * kBS];
  const int W = w.W, H = w.H, slab_h = w.slab_h ? w.slab_h : H;
  const int x0 = blockIdx.x * 32, y0 = blockIdx.y * 32;
  const int ly = threadIdx.x >> 3, lx = (threadIdx.x & 7) * 4;
  const int x = x0 + lx, y = y0 + ly;
  const bool in = x < W && y < H;
  const int slab = y / slab_h, ys = y - slab * slab_h;
  const int64_t i = (int64_t)y * W + x, N = (int64_t)slab_h * W;
  int l[4] = {kLake, kLake, kLake, kLake};
  if (in) {
    const int* first = w.state + slab * N;
    int c[4];
    if ((W & 3) == 0) {
      const int4 v = *reinterpret_cast<const int4*>(w.state + i);
      c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++) c[k] = x + k < W ? w.state[i + k] : label_code(kLake);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) c[k] = resolve(c[k], w.bstate);  // all in flight at once
#pragma unroll
    for (int k = 0; k < 4; k++) l[k] = decode_label(c[k], first, w.bstate, stuck);
  }
  *reinterpret_cast<int4*>(&L[(ly + 1) * kBS + 4 + lx]) =
      make_int4(border_key(l[0]), border_key(l[1]), border_key(l[2]), border_key(l[3]));
  if (threadIdx.x < 132) {
    int hx, hy;
    halo_cell(threadIdx.x, hx, hy);
    const int gx = x0 + hx, gy = y0 + hy;
    int key = kNoLabel;
    if (gx >= 0 && gx < W && gy >= 0 && gy < H)
      key = border_key(decode_label(w.bstate[border_index(gx, gy, w.tiles_x)],
                                    w.state + (gy / slab_h) * N, w.bstate, stuck));
    L[(hy + 1) * kBS + 4 + hx] = key;
  }
  __syncthreads();
  if (!in) return;
  const int64_t is = (int64_t)ys * W + x;
  if (!last || *real + (uint32_t)slab == *last) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (x + k < W) label[is + k] = l[k];
  }
  if (gate && gate[slab]) return;
  const unsigned int b = border_of_4(L, lx, ly, ys > 0, ys < slab_h - 1);
#pragma unroll
  for (int k = 0; k < 4; k++)
    if ((b >> k & 1u) && x + k < W) atomicAdd(&count[is + k], 1u);
}

cageo_status border_u32_from_state(const TraceWork& w, int* label, uint32_t* count,
                                   const int* gate, int mode, const uint32_t* real,
                                   const uint32_t* last, cudaStream_t s) {
  border_state_kernel<<<dim3(w.tiles_x, w.tiles_y), 256, 0, s>>>(
      w, label, count, gate, mode == CAGEO_TRACE_DEAD_END_ERROR ? kError : 0, real, last);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

cageo_status border_float(const int* label, float* count, int W, int H, cudaStream_t s) {
  const dim3 g((W + 31) / 32, (H + 31) / 32);
  border_kernel<float><<<g, 256, 0, s>>>(label, count, W, H);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

}  // namespace cageo

using namespace cageo;

extern "C" size_t cageo_trace_workspace_size(int W, int H) {
  if (!valid_dims(W, H)) return 0;
  return trace_workspace_bytes(W, H);
}

extern "C" cageo_status cageo_trace_mode(const int8_t* d_dir, const float* d_streams,
                                         int* d_label, int W, int H, int mode,
                                         void* d_workspace, size_t workspace_bytes,
                                         cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_dir && d_streams && d_label && valid_dims(W, H), "pointers and size");
  CAGEO_CHECK_ARG(mode == CAGEO_TRACE_CPU_COMPAT || mode == CAGEO_TRACE_DEAD_END_ERROR,
                  "tracing mode");
  Scratch ws;
  cageo_status st = ws.acquire(d_workspace, workspace_bytes, trace_workspace_bytes(W, H), stream);
  if (st) return st;
  TraceWork w = trace_carve(ws.ptr, W, H);
  if ((st = trace_run(d_dir, d_streams, nullptr, d_label, w, stream, mode, true))) return st;
  CAGEO_CUDA(cudaStreamSynchronize(stream));
  return trace_check_status(w, nullptr);
}

extern "C" cageo_status cageo_trace(const int8_t* d_dir, const float* d_streams,
                                    int* d_label, int W, int H, void* d_workspace,
                                    size_t workspace_bytes, cudaStream_t stream) {
  return cageo_trace_mode(d_dir, d_streams, d_label, W, H, CAGEO_TRACE_CPU_COMPAT, d_workspace,
                          workspace_bytes, stream);
}

extern "C" cageo_status cageo_border_accumulate(const int* d_label, float* d_count, int W,
                                                int H, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_label && d_count && valid_dims(W, H), "pointers and size");
  return border_float(d_label, d_count, W, H, stream);
}
