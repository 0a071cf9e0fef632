// routing.cu -- A7 D8 flow routing with the reference CPU path's rules
// (src/flowrouting/FlowRoutingAlgorithmCPUOpenMP.h:53-249).
//
// First pass: border cells point outward (corners diagonally), cells equal to
// 0 are streams (flatDist -2, no direction), others take the steepest
// strictly-descending neighbour in N, NE, E, SE, S, SW, W, NW order with
// diagonal drops divided by 1.41421356f, the first maximum winning.  Cells
// with no descending neighbour are flat.
//
// Flats: the reference assigns layer k = 1, 2, ... to flat cells that have a
// neighbour in layer k-1 (layer 0 = cells with a direction, flatDist -1)
// whose elevation is <= theirs, taking the direction of the LAST such
// neighbour in N..NW order.  A flat cell has no lower neighbour, so such a
// neighbour is at its own elevation, and adjacent flat cells are level with
// each other: layers 1 need the elevations once (the first pass finds them,
// with their directions), all later layers only the masks of flat cells.  (A
// NaN cell is level with nothing and is left out of the masks.)
// Layer numbers are breadth-first distances; they are computed tile by tile
// (32x32) from three things only: the tile's mask of flat cells, its mask of
// layer-1 cells, and the distances on the neighbouring tiles' rims, kept in a
// compact array (4 sides x 32 per tile).  A visit of the distance flood so
// moves 0.8 KB, against 9 KB when it staged distances and elevations, and
// writes back changed rims.  When the rims are final, one pass over the tiles
// recomputes the distances inside and applies the last-match rule.
//
// The GPU-order mode follows the reference's GPU routing instead
// (src/flowrouting/FlowRoutingAlgorithmGPUCUDAOriginal.cu:200-271 and
// :391-437): NODATA cells get flatDist -3 and are skipped as neighbours;
// layer 1 may drain into any cell with a negative flatDist (streams too)
// whose non-NODATA elevation is <= the flat cell's; a later layer k drains
// into a cell of an earlier layer; the FIRST match in the order N, W, E,
// S, NW, NE, SW, SE wins.  The layer numbers are again BFS distances (and a
// stream, at 0, is never level with a flat cell: one above 0 has a direction,
// one below 0 is lower).
#include <algorithm>
#include <type_traits>
#include "common.cuh"
#include "routing.cuh"
#include "stage_math.cuh"
#include "tilequeue.cuh"

namespace cageo {

constexpr int kFlatInf = 0x3fffffff;
enum : int { R_NFLAT = 0, R_ERR = 3, R_US_BFS = 8, R_PASSES = 9,
             R_TILES = 10, R_KCYC_LOAD = 11, R_KCYC_BFS = 12, R_KCYC_STORE = 13,
             R_BAR_COUNT = kBarCountSlot, R_BAR_GEN = kBarGenSlot,
             R_HEAD = 128,     // work-queue tickets handed out (own 128-byte line)
             R_TAIL = 160,     // work-queue entries pushed (own line)
             R_DONE = 192,     // tiles finished (own line)
             R_SIZE = kRouteScalars };
constexpr int kFT = 32;          // flat tile size
constexpr int kFWarps = 32;      // most warps per block of the distance flood
enum : int { kRTop = 0, kRBottom = 1, kRLeft = 2, kRRight = 3 };
constexpr int kRimCells = 4 * kFT;

size_t route_workspace_bytes(int W, int H) {
  const size_t nt = (size_t)((W + kFT - 1) / kFT) * ((H + kFT - 1) / kFT);
  return align_up(nt, 256) + align_up(nt * 4, 256) + align_up((2 * nt + kRingSlack) * 4, 256) +
         2 * align_up(nt * kFT * 4, 256) + align_up(nt * kRimCells * 4, 256) +
         align_up(R_SIZE * 4, 256);
}

RouteWork route_carve(void* base, int W, int H) {
  RouteWork w;
  w.W = W;
  w.H = H;
  w.tiles_x = (W + kFT - 1) / kFT;
  w.tiles_y = (H + kFT - 1) / kFT;
  const size_t nt = (size_t)w.tiles_x * w.tiles_y;
  char* p = (char*)base;
  w.tflat = (uint8_t*)p;
  p += align_up(nt, 256);
  w.queued = (int*)p;
  p += align_up(nt * 4, 256);
  w.lists = (int*)p;
  p += align_up((2 * nt + kRingSlack) * 4, 256);
  w.mflat = (uint32_t*)p;
  p += align_up(nt * kFT * 4, 256);
  w.mfirst = (uint32_t*)p;
  p += align_up(nt * kFT * 4, 256);
  w.rim = (int*)p;
  p += align_up(nt * kRimCells * 4, 256);
  w.scal = (unsigned int*)p;
  return w;
}

// x / 1.41421356237309505f, correctly rounded for magnitudes in (1e-30, 1e30):
// the product with the rounded reciprocal and one correction by its residue
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990); equal to the division for every mantissa (checked over
// all 2^24 floats of [1, 4)).  3 instructions against ~10.
__device__ __forceinline__ float div_sqrt2(float x) {
  constexpr float kS = 1.41421356237309505f, kR = 1.0f / kS;
  const float q = __fmul_rn(x, kR);
  return __fmaf_rn(__fmaf_rn(-q, kS, x), kR, q);
}

// The steepest descent from c to its neighbours v in N, NE, E, SE, S, SW, W, NW
// order, diagonal drops divided by sqrt(2), the first maximum winning: its
// index, or 8 where no neighbour is lower.  GPU: NODATA neighbours are skipped.
// All eight slopes at once, their maximum, then the first equal to it: ~45
// instructions, against ~75 for a running maximum.
template <bool GPU>
__device__ __forceinline__ int steepest_of(float c, const float (&v)[8], float nodata) {
  float s[8];
#pragma unroll
  for (int n = 0; n < 8; n++) s[n] = GPU && v[n] == nodata ? 0.0f : __fsub_rn(c, v[n]);
  const float diag = fmaxf(fmaxf(s[1], s[3]), fmaxf(s[5], s[7]));
  if (diag > 0.0f && !(diag > 1e-30f && diag < 1e30f)) {
    // Outside the quick division's range: the largest diagonal drop decides
    // (a smaller one that rounds to the same quotient is in range with it).
    float best = 0.0f;
    int got = 8;
#pragma unroll
    for (int n = 0; n < 8; n++) {
      const float d = n & 1 ? __fdiv_rn(s[n], 1.41421356237309505f) : s[n];
      if (d > best) {
        best = d;
        got = n;
      }
    }
    return got;
  }
#pragma unroll
  for (int n = 1; n < 8; n += 2) s[n] = div_sqrt2(s[n]);
  const float best = fmaxf(fmaxf(fmaxf(s[0], s[2]), fmaxf(s[4], s[6])),
                           fmaxf(fmaxf(s[1], s[3]), fmaxf(s[5], s[7])));
  int got = 8;
#pragma unroll
  for (int n = 7; n >= 0; n--)
    if (s[n] == best) got = n;
  return best > 0.0f ? got : 8;
}

// Direction n as (dx, dy) bytes; n = 8: none.
__device__ __forceinline__ unsigned int d8_dir(int n) {
  const unsigned int dx = __byte_perm(0x01010100u, 0xffffff00u, n);
  const unsigned int dy = __byte_perm(0x0100ffffu, 0xff000101u, n);
  return n < 8 ? __byte_perm(dx, dy, 0x0040u) & 0xffffu : 0u;
}

// Staged elevations of a tile and the two cells around it: rows y0 - 2 ..
// y0 + 33, columns x0 - 4 .. x0 + 35 (x0 - 2 .. x0 + 33 are used), so that the
// tile's own columns start on a 16-byte boundary.
constexpr int kES = 40;

// Whether the cell at staged position (sx, sy) -- column gx, in the grid if
// `in`, row ys of its slab -- has a direction from the first pass.
template <bool GPU>
__device__ __forceinline__ bool has_direction(const float* E, int sx, int sy, bool in, int gx,
                                              int ys, int W, int slab_h, float nodata) {
  if (!in) return false;
  if (gx == 0 || gx == W - 1 || ys == 0 || ys == slab_h - 1) return true;
  const float* e = E + sy * kES + sx;
  const float c = *e;
  if (c == 0.0f || (GPU && c == nodata)) return false;
  float m = kInf;
#pragma unroll
  for (int n = 0; n < 8; n++) {
    const float v = e[d8_dy(n) * kES + d8_dx(n)];
    if (!(GPU && v == nodata)) m = fminf(m, v);
  }
  return m < c;
}

// First pass: directions, the masks of flat and of layer-1 cells with the
// directions of the latter, the rims' first distances, and (fd not null) the
// flat distances known so far.  A block of 8 warps per 32x32 tile, a warp per
// 4 rows (lane = column): the three elevations of a row serve three rows of
// outputs from registers.  A layer-1 cell needs to know which neighbours have
// a direction, so the ring around the tile is decided too (132 cells).
template <bool GPU>
__global__ void __launch_bounds__(256) d8_kernel(const float* __restrict__ dem,
                                                 char2* __restrict__ dir,
                                                 int* __restrict__ fd, RouteWork w, float nodata) {
  const int W = w.W, H = w.H;
  const int slab_h = w.slab_h ? w.slab_h : H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x0 = blockIdx.x * kFT, y0 = blockIdx.y * kFT;
  __shared__ __align__(16) float E[36 * kES];
  __shared__ unsigned int Hd[34];       // cells with a direction, rows -1..32, columns 0..31
  __shared__ unsigned int Hl, Hr, Hc;   // columns -1 and 32 (bit = row 0..31), corners
  __shared__ unsigned int F[kFT], S[kFT];
  if ((W & 3) == 0 && x0 + kFT <= W && ((uintptr_t)dem & 15u) == 0) {
    // The tile's columns by 16-byte copies, the two beside them on either side
    // by 4-byte ones: 432 copies instead of 1296.
    for (int k = threadIdx.x; k < 36 * 8 + 36 * 4; k += 256) {
      const bool mid = k < 36 * 8;
      const int j = k - 36 * 8;
      const int sy = mid ? k >> 3 : j >> 2;
      const int sx = mid ? 4 + 4 * (k & 7) : (j & 2 ? 36 : 2) + (j & 1);
      const int gx = x0 - 4 + sx, gy = y0 - 2 + sy;
      float* e = &E[sy * kES + sx];
      if (gy >= 0 && gy < H && gx >= 0 && gx < W) {
        if (mid) cp_async16(e, dem + (int64_t)gy * W + gx);
        else cp_async4(e, dem + (int64_t)gy * W + gx);
      }
    }
  } else {
    for (int k = threadIdx.x; k < 36 * 36; k += 256) {
      const int sy = k / 36, sx = k - sy * 36 + 2;
      const int gx = x0 - 4 + sx, gy = y0 - 2 + sy;
      if (gx >= 0 && gx < W && gy >= 0 && gy < H)
        cp_async4(&E[sy * kES + sx], dem + (int64_t)gy * W + gx);
    }
  }
  cp_async_wait();
  __syncthreads();
  const int x = x0 + lane, yw = y0 + 4 * warp;  // this warp's first row
  const bool xin = x < W, xborder = x == 0 || x == W - 1;
  const int ys0 = yw % slab_h;  // its row in its slab
  // Row of the slab `k` rows further (k < 37).
  auto slab_row = [&](int k) {
    int ys = ys0 + k;
    while (ys >= slab_h) ys -= slab_h;
    return ys;
  };
  // A tile of interior cells only needs no test of the border or the grid.
  const int top = y0 % slab_h;
  const bool plain = x0 > 0 && x0 + kFT < W && top > 0 && top + kFT < slab_h && y0 + kFT <= H;
  // 0..7: direction; 8: flat (| the level neighbours << 4, a bit per direction);
  // 9: border; 10: stream, NODATA or outside
  int code[4];
  auto directions = [&](auto interior) {
    constexpr bool kPlain = decltype(interior)::value;
    const float* e = E + (4 * warp + 1) * kES + lane + 3;  // row above this warp's first
    float a0 = e[0], a1 = e[1], a2 = e[2];
    float b0 = e[kES], b1 = e[kES + 1], b2 = e[kES + 2];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float* r = e + (k + 2) * kES;
      const float c0 = r[0], c1 = r[1], c2 = r[2];
      const float v[8] = {a1, a2, b2, c2, c1, c0, b0, a0};
      int n = steepest_of<GPU>(b1, v, nodata);
      if (b1 == 0.0f || (GPU && b1 == nodata)) n = 10;
      if constexpr (!kPlain) {
        const int ys = slab_row(k);
        if (xborder || ys == 0 || ys == slab_h - 1) n = 9;
        if (!xin || yw + k >= H) n = 10;
      }
      // (CPU rules: a NaN cell is flat, but level with nothing, so that no layer
      // enters or leaves it; the GPU order compares elevations for layer 1 only.)
      const unsigned int f = __ballot_sync(0xffffffffu, n == 8 && (GPU || b1 == b1));
      const unsigned int h = __ballot_sync(0xffffffffu, kPlain ? n < 8 : n < 8 || n == 9);
      code[k] = n;
      if (f) {  // (no neighbour is lower: <= is level)
        int level = 0;
#pragma unroll
        for (int d = 0; d < 8; d++)
          if (v[d] <= b1 && !(GPU && v[d] == nodata)) level |= 16 << d;
        if (n == 8) code[k] |= level;
      }
      if (lane == 0) {
        Hd[4 * warp + k + 1] = h;
        F[4 * warp + k] = f;
      }
      a0 = b0; a1 = b1; a2 = b2;
      b0 = c0; b1 = c1; b2 = c2;
    }
  };
  if (plain) directions(std::true_type());
  else directions(std::false_type());
  // The ring: rows -1 and 32 (warps 0, 1), columns -1 and 32 (2, 3), corners.
  if (warp < 5) {
    const bool col = warp == 2 || warp == 3, corner = warp == 4;
    const int rx = corner ? (lane & 1 ? 32 : -1) : col ? (warp == 2 ? -1 : 32) : lane;
    const int ry = corner ? (lane & 2 ? 32 : -1) : col ? lane : (warp ? 32 : -1);
    const int gx = x0 + rx, gy = y0 + ry;
    const bool in = (!corner || lane < 4) && gx >= 0 && gx < W && gy >= 0 && gy < H;
    const unsigned int h = __ballot_sync(
        0xffffffffu, has_direction<GPU>(E, rx + 4, ry + 2, in, gx, in ? gy % slab_h : 0, W,
                                        slab_h, nodata));
    if (lane == 0) {
      if (warp == 2) Hl = h;
      else if (warp == 3) Hr = h;
      else if (warp == 4) Hc = h;
      else Hd[warp ? 33 : 0] = h;
    }
  }
  __syncthreads();
  // Directions; flat cells look for a level neighbour with a direction.
  int nflat = 0;
  // Bits 0..2: the cells at x - 1, x, x + 1 of row r (0..33 for rows -1..32)
  // that have a direction.
  auto row3 = [&](int r) {
    const unsigned int h = Hd[r];
    const unsigned int l = r == 0 ? Hc : r == 33 ? Hc >> 2 : Hl >> (r - 1);
    const unsigned int g = r == 0 ? Hc >> 1 : r == 33 ? Hc >> 3 : Hr >> (r - 1);
    return __funnelshift_r((h << 1) | (l & 1u), (h >> 31) | ((g & 1u) << 1), lane) & 7u;
  };
  unsigned int gn = row3(4 * warp), gm = row3(4 * warp + 1);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int ty = 4 * warp + k, y = y0 + ty;
    const unsigned int gs = row3(ty + 2);
    int n = code[k] & 15;
    bool first = false;
    if (n == 8) {
      nflat++;
      // 8 bits in N..NW order: level neighbours with a direction.
      const unsigned int m = ((gn >> 1 & 3u) | (gm & 4u) | (gs & 4u) << 1 | (gs & 2u) << 3 |
                              (gs & 1u) << 5 | (gm & 1u) << 6 | (gn & 1u) << 7) &
                             (unsigned int)code[k] >> 4;
      first = m != 0;
      if (GPU) {
        constexpr int order[8] = {0, 6, 2, 4, 7, 1, 5, 3};  // N W E S NW NE SW SE as D8 indices
#pragma unroll
        for (int j = 7; j >= 0; j--)
          if (m >> order[j] & 1u) n = order[j];
      } else if (first) {
        n = 31 - __clz(m);  // the last in D8 order
      }
    }
    gn = gm;
    gm = gs;
    const unsigned int s = __ballot_sync(0xffffffffu, first);
    if (lane == 0) S[ty] = s;
    if (!xin || y >= H) continue;
    const int64_t i = (int64_t)y * W + x;
    unsigned int d = d8_dir(n);
    if (n == 9) {
      const int ys = slab_row(k);
      const int dx = x == 0 ? -1 : x == W - 1 ? 1 : 0, dy = ys == 0 ? -1 : ys == slab_h - 1 ? 1 : 0;
      d = (dx & 0xff) | (dy & 0xff) << 8;
    }
    reinterpret_cast<unsigned short*>(dir)[i] = (unsigned short)d;
    if (fd) {
      // Flat cells beyond layer 1 start unresolved (0).
      fd[i] = (code[k] & 15) == 8 ? (first ? 1 : 0)
              : code[k] != 10 ? -1
              : (GPU && E[(ty + 2) * kES + lane + 4] != 0.0f) ? -3 : -2;
    }
  }
  nflat = __reduce_add_sync(0xffffffffu, nflat);
  __syncthreads();
  const int t = blockIdx.y * w.tiles_x + blockIdx.x;
  if (lane == 0 && nflat) atomicAdd(&w.scal[R_NFLAT], (unsigned int)nflat);  // statistics only
  if (warp == 4) {
    const unsigned int f = F[lane], s = S[lane];
    w.mflat[t * kFT + lane] = f;
    w.mfirst[t * kFT + lane] = s;
    const bool more = __any_sync(0xffffffffu, (f & ~s) != 0);
    if (lane == 0) w.tflat[t] = more;
  } else if (warp < 4) {
    // Rim entries: 0 not flat, 1 layer 1, infinite otherwise.
    const int rx = warp == kRLeft ? 0 : warp == kRRight ? 31 : lane;
    const int ry = warp == kRTop ? 0 : warp == kRBottom ? 31 : lane;
    const bool f = F[ry] >> rx & 1u, s = S[ry] >> rx & 1u;
    w.rim[(size_t)t * kRimCells + warp * kFT + lane] = s ? 1 : f ? kFlatInf : 0;
  }
}

// ---- distances ------------------------------------------------------------
// The flat BFS's queue (tilequeue.cuh): tile states in w.queued, the ring
// in w.lists.
__device__ __forceinline__ TileQueue route_queue(const RouteWork& w) {
  return TileQueue{w.queued,
                   w.lists,
                   2u * (unsigned int)(w.tiles_x * w.tiles_y) + kRingSlack,
                   w.scal + R_HEAD,
                   w.scal + R_TAIL,
                   w.scal + R_DONE,
                   (int*)(w.scal + R_ERR)};
}

// Per-warp visit statistics (lane 0), flushed every 64 visits and at the end.
struct FlatStats {
  unsigned int tiles = 0, kload = 0, kbfs = 0, kstore = 0;
};

__device__ __forceinline__ void flush_flat_stats(const RouteWork& w, FlatStats& st) {
  if (!st.tiles) return;
  atomicAdd(&w.scal[R_TILES], st.tiles);
  atomicAdd(&w.scal[R_KCYC_LOAD], st.kload);
  atomicAdd(&w.scal[R_KCYC_BFS], st.kbfs);
  atomicAdd(&w.scal[R_KCYC_STORE], st.kstore);
  st = FlatStats{};
}

// The rim entries around a tile: cells next to its top, bottom, left and right
// side, corners in lanes 0..3 (TL, TR, BL, BR).  L2: other SMs write them.
struct FlatHalo {
  int t, b, l, r, c;
};

__device__ __forceinline__ FlatHalo flat_halo(const RouteWork& w, int t, int lane) {
  const int tx = t % w.tiles_x, ty = t / w.tiles_x;
  const bool up = ty > 0, dn = ty + 1 < w.tiles_y, lf = tx > 0, rt = tx + 1 < w.tiles_x;
  auto at = [&](bool in, int tile, int side, int k) {
    return in ? __ldcg(w.rim + (size_t)tile * kRimCells + side * kFT + k) : 0;
  };
  FlatHalo h;
  h.t = at(up, t - w.tiles_x, kRBottom, lane);
  h.b = at(dn, t + w.tiles_x, kRTop, lane);
  h.l = at(lf, t - 1, kRRight, lane);
  h.r = at(rt, t + 1, kRLeft, lane);
  const bool cdn = lane & 2, crt = lane & 1;
  h.c = at(lane < 4 && (cdn ? dn : up) && (crt ? rt : lf),
           t + (cdn ? w.tiles_x : -w.tiles_x) + (crt ? 1 : -1), cdn ? kRTop : kRBottom,
           crt ? 0 : 31);
  return h;
}

// Levels the halo gives this lane's cells of the four sides (top and bottom:
// lane = column; left and right: lane = row): 1 + the least distance of the
// flat cells next to it outside the tile.
struct FlatSeeds {
  int t, b, l, r;
};

__device__ __forceinline__ FlatSeeds flat_seeds(const FlatHalo& h, unsigned int flat, int lane) {
  auto dist = [](int v) { return v == 0 ? kFlatInf : v; };  // not flat: no distance
  const int c = dist(h.c);
  const int tl = __shfl_sync(0xffffffffu, c, 0), tr = __shfl_sync(0xffffffffu, c, 1);
  const int bl = __shfl_sync(0xffffffffu, c, 2), br = __shfl_sync(0xffffffffu, c, 3);
  auto near = [&](int v, int lo, int hi, bool is_flat) {
    const int u = __shfl_up_sync(0xffffffffu, v, 1), d = __shfl_down_sync(0xffffffffu, v, 1);
    const int m = min(v, min(lane == 0 ? lo : u, lane == 31 ? hi : d));
    return is_flat && m < kFlatInf ? m + 1 : kFlatInf;
  };
  const unsigned int f0 = __shfl_sync(0xffffffffu, flat, 0), f31 = __shfl_sync(0xffffffffu, flat, 31);
  FlatSeeds s;
  s.t = near(dist(h.t), tl, tr, f0 >> lane & 1u);
  s.b = near(dist(h.b), bl, br, f31 >> lane & 1u);
  s.l = near(dist(h.l), tl, bl, flat & 1u);
  s.r = near(dist(h.r), tr, br, flat >> 31);
  return s;
}

// Distances inside a tile by a bit-parallel breadth-first search: lane y holds
// row y as a bit mask.  Levels are visited in increasing order, one dilation
// each, so the first level that reaches a cell is its distance: step(front, L)
// gets the cells of each level.  Four levels between two looks whether the
// front has died out (the search then jumps to the next level that has seeds);
// every(L) is called there, before levels L .. L + 3.
template <class Every, class Step>
__device__ __forceinline__ void flat_levels(unsigned int flat, unsigned int first,
                                            const FlatSeeds& sd, int lane, Every every, Step step) {
  auto next_level = [&](int after) {  // least seed level above `after`
    int m = kFlatInf;
    if (sd.t > after) m = min(m, sd.t);
    if (sd.b > after) m = min(m, sd.b);
    if (sd.l > after) m = min(m, sd.l);
    if (sd.r > after) m = min(m, sd.r);
    if (first && after < 1) m = min(m, 1);
    return __reduce_min_sync(0xffffffffu, m);
  };
  int L = next_level(0);
  unsigned int open = flat, front = 0;
  for (int guard = 0; guard < 4 * kFT * kFT && L < kFlatInf; guard++) {
    every(L);
#pragma unroll
    for (int k = 0; k < 4; k++, L++) {
      const unsigned int tb = __ballot_sync(0xffffffffu, sd.t == L);
      const unsigned int bb = __ballot_sync(0xffffffffu, sd.b == L);
      unsigned int seeds = (L == 1 ? first : 0u) | (sd.l == L ? 1u : 0u) |
                           (sd.r == L ? 0x80000000u : 0u);
      if (lane == 0) seeds |= tb;
      if (lane == kFT - 1) seeds |= bb;
      unsigned int up = __shfl_up_sync(0xffffffffu, front, 1);
      unsigned int dn = __shfl_down_sync(0xffffffffu, front, 1);
      if (lane == 0) up = 0;
      if (lane == kFT - 1) dn = 0;
      const unsigned int v = front | up | dn;
      front = ((v | (v << 1) | (v >> 1)) | seeds) & open;
      open &= ~front;
      step(front, L);
    }
    if (!__any_sync(0xffffffffu, front != 0)) {
      if (!__any_sync(0xffffffffu, open != 0)) break;
      L = next_level(L - 1);
    }
  }
}

// Every reached cell's distance to emit(x, level) (this lane's row).  The
// levels are kept as offsets from a base in 6 bit planes and handed over once
// per segment of at most 64 consecutive levels.
template <class Emit>
__device__ __forceinline__ void flat_bfs(unsigned int flat, unsigned int first, const FlatSeeds& sd,
                                         int lane, Emit emit) {
  int base = 0, after = 0;  // the segment's levels: base .. after - 1
  unsigned int seg = 0, p0 = 0, p1 = 0, p2 = 0, p3 = 0, p4 = 0, p5 = 0;
  auto flush = [&]() {
    for (unsigned int r = seg; r; r &= r - 1) {
      const int x = __ffs(r) - 1;
      const int off = ((p0 >> x) & 1) | (((p1 >> x) & 1) << 1) | (((p2 >> x) & 1) << 2) |
                      (((p3 >> x) & 1) << 3) | (((p4 >> x) & 1) << 4) | (((p5 >> x) & 1) << 5);
      emit(x, base + off);
    }
    seg = p0 = p1 = p2 = p3 = p4 = p5 = 0;
  };
  flat_levels(flat, first, sd, lane,
              [&](int L) {
                if (L != after || L - base == 64) {
                  flush();
                  base = L;
                }
                after = L + 4;
              },
              [&](unsigned int front, int L) {
                const int off = L - base;  // 0..63
                seg |= front;
                if (off & 1) p0 |= front;
                if (off & 2) p1 |= front;
                if (off & 4) p2 |= front;
                if (off & 8) p3 |= front;
                if (off & 16) p4 |= front;
                if (off & 32) p5 |= front;
              });
  flush();
  __syncwarp();
}

// One visit: the distances on the tile's rim for its halo.  A neighbour is
// queued only when a rim cell that fell is more than one step below a flat
// cell next to it (distances only fall, so what holds for the staged ones
// holds for the present ones).
__device__ void flat_tile(const RouteWork& w, int t, int lane, FlatStats& st) {
  const long long c0 = clock64();
  int* own = w.rim + (size_t)t * kRimCells + lane;
  const unsigned int flat = w.mflat[t * kFT + lane], first = w.mfirst[t * kFT + lane];
  const FlatHalo h = flat_halo(w, t, lane);
  const int oT = __ldcg(own + kRTop * kFT), oB = __ldcg(own + kRBottom * kFT);
  const int oL = __ldcg(own + kRLeft * kFT), oR = __ldcg(own + kRRight * kFT);
  const bool visited = ((volatile uint8_t*)w.tflat)[t] == 2;
  const FlatSeeds sd = flat_seeds(h, flat, lane);
  const long long c1 = clock64();
  long long c2 = c1;
  unsigned int want = 0;  // neighbours to queue: 1 L, 2 R, 4 T, 8 B, 16 TL, 32 TR, 64 BL, 128 BR
  const bool lower = sd.t < oT || sd.b < oB || sd.l < oL || sd.r < oR;
  if (!visited || __any_sync(0xffffffffu, lower)) {
    // Only the rim's distances are wanted: each lane notes the level that
    // reaches its cell of each side.
    int nT = kFlatInf, nB = kFlatInf, nL = kFlatInf, nR = kFlatInf;
    flat_levels(flat, first, sd, lane, [](int) {}, [&](unsigned int front, int L) {
      const unsigned int top = __shfl_sync(0xffffffffu, front, 0);
      const unsigned int bottom = __shfl_sync(0xffffffffu, front, 31);
      if (top >> lane & 1u) nT = L;
      if (bottom >> lane & 1u) nB = L;
      if (front & 1u) nL = L;
      if (front >> 31) nR = L;
    });
    c2 = clock64();
    if (!visited && lane == 0) w.tflat[t] = 2;
    auto side = [&](int which, int v, int o, int hv, unsigned int bit, int clo, int chi,
                    unsigned int lobit, unsigned int hibit) {
      const bool fell = v < o;
      if (!__any_sync(0xffffffffu, fell)) return;
      if (fell) own[which * kFT] = v;
      const int u = __shfl_up_sync(0xffffffffu, hv, 1), d = __shfl_down_sync(0xffffffffu, hv, 1);
      if (__any_sync(0xffffffffu, fell && v + 1 < max(hv, max(u, d)))) want |= bit;
      const int lo = __shfl_sync(0xffffffffu, h.c, clo), hi = __shfl_sync(0xffffffffu, h.c, chi);
      const unsigned int at = __ballot_sync(0xffffffffu, fell && v + 1 < (lane == 0 ? lo : hi));
      if (at & 1u) want |= lobit;
      if (at >> 31) want |= hibit;
    };
    side(kRTop, nT, oT, h.t, 4u, 0, 1, 16u, 32u);
    side(kRBottom, nB, oB, h.b, 8u, 2, 3, 64u, 128u);
    side(kRLeft, nL, oL, h.l, 1u, 0, 2, 16u, 64u);
    side(kRRight, nR, oR, h.r, 2u, 1, 3, 32u, 128u);
    // The rims are visible before any neighbour is queued or the tile's state
    // changes.
    __threadfence();
    __syncwarp();
    if (want) {
      // (A side is wanted only where a neighbour lies: outside the grid the
      // staged entries are 0.)
      const int dx = lane == 1 || lane == 5 || lane == 7 ? -1 : lane == 2 || lane == 6 || lane == 8 ? 1 : 0;
      const int dy = lane == 3 || lane == 5 || lane == 6 ? -1 : lane == 4 || lane == 7 || lane == 8 ? 1 : 0;
      const int n = t + dy * w.tiles_x + dx;
      const bool go = lane >= 1 && lane < 9 && (want >> (lane - 1) & 1u);
      tq_enqueue(route_queue(w), go && ((volatile uint8_t*)w.tflat)[n], n);
    }
  }
  if (lane == 0) {
    const long long c3 = clock64();
    st.tiles++;
    st.kload += (unsigned int)((c1 - c0) >> 10);
    st.kbfs += (unsigned int)((c2 - c1) >> 10);
    st.kstore += (unsigned int)((c3 - c2) >> 10);
  }
}

// The distance flood: every tile with flat cells beyond layer 1 is queued, one
// 2x2 parity class of tiles after another (grid barrier between), so tiles
// searched at the same time are rarely neighbours and each class starts from
// the finished rims of the classes before it; then the warps drain the
// asynchronous queue (tilequeue.cuh).  No pass barriers: a free warp takes the
// next queued tile at once.  Waits are bounded; a limit sets the error flag.
__global__ void __launch_bounds__(kFWarps * 32, 1) flat_relax_kernel(RouteWork w) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int ntiles = w.tiles_x * w.tiles_y;
  GridSync gs{w.scal + R_BAR_COUNT, w.scal + R_BAR_GEN, (int*)(w.scal + R_ERR)};
  volatile unsigned int* vs = w.scal;
  const TileQueue q = route_queue(w);
  unsigned long long t0;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  const int gwarp = blockIdx.x * warps + warp, nwarps = gridDim.x * warps;
  bool go = true;
  for (int c = 0; c < 4 && go; c++) {
    for (int base = gwarp * 32; base < ntiles; base += nwarps * 32) {
      const int i = base + lane, tx = i % w.tiles_x, ty = i / w.tiles_x;
      tq_enqueue(q, i < ntiles && ((tx & 1) | ((ty & 1) << 1)) == c && w.tflat[i], i);
    }
    go = grid_barrier(gs, gridDim.x);
  }
  FlatStats st;
  if (go) {
    const unsigned int visit_cap = 1000u * (unsigned int)min(ntiles, 4000000);
    long long ticket = -1;
    unsigned int ns = 32, finished = 0;
    for (long long idle = 0;; idle++) {
      int t = -1;
      if (lane == 0) t = tq_try_dequeue(q, &ticket);
      t = __shfl_sync(0xffffffffu, t, 0);
      __syncwarp();  // lane 0's fence holds for the loads of all lanes (a shuffle orders no memory)
      if (t >= 0) {
        flat_tile(w, t, lane, st);
        if (lane == 0) {
          tq_finish(q, t);
          finished++;
          if (st.tiles >= 64) flush_flat_stats(w, st);
        }
        __syncwarp();
        idle = 0;
        ns = 32;
        continue;
      }
      int end = 0;
      if (lane == 0) {
        if (tq_drained(q, &finished) || vs[R_ERR]) end = 1;
        else if (idle > (1LL << 25) || vs[R_TILES] > visit_cap) end = 2;
      }
      end = __shfl_sync(0xffffffffu, end, 0);
      if (end) {
        if (lane == 0 && end == 2) atomicCAS((int*)(w.scal + R_ERR), 0, 2);
        break;
      }
      __nanosleep(ns);
      if (ns < 512) ns <<= 1;
    }
  }
  if (lane == 0) flush_flat_stats(w, st);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    unsigned long long t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
    vs[R_PASSES] = 1u;  // one drain of the queue
    vs[R_US_BFS] = (unsigned int)((t1 - t0) / 1000);
  }
}

// Directions (and, fd not null, flatDist) of the flat cells beyond layer 1,
// one warp per tile that holds any: the distances inside from the final rims,
// then, lane = column, a row at a time: CPU rules: the LAST neighbour in N..NW
// order in the previous layer; GPU order: the FIRST neighbour in N, W, E, S,
// NW, NE, SW, SE order in an earlier layer (which is the previous one).
constexpr int kDS = 35;  // row stride of the staged distances (34 used)
constexpr int kDirWarps = 8;
template <bool GPU>
__global__ void __launch_bounds__(kDirWarps * 32) flat_dir_kernel(char2* __restrict__ dir,
                                                                  int* __restrict__ fd, RouteWork w) {
  __shared__ int Ds[kDirWarps][34 * kDS];
  const int lane = threadIdx.x & 31, t = blockIdx.x * kDirWarps + (threadIdx.x >> 5);
  if (t >= w.tiles_x * w.tiles_y || !w.tflat[t]) return;
  int* D = Ds[threadIdx.x >> 5];
  const unsigned int flat = w.mflat[t * kFT + lane], first = w.mfirst[t * kFT + lane];
  const FlatHalo h = flat_halo(w, t, lane);
  const FlatSeeds sd = flat_seeds(h, flat, lane);
#pragma unroll 8
  for (int y = 0; y < kFT; y++) D[(y + 1) * kDS + lane + 1] = 0;  // 0: no distance
  D[lane + 1] = h.t;
  D[33 * kDS + lane + 1] = h.b;
  D[(lane + 1) * kDS] = h.l;
  D[(lane + 1) * kDS + 33] = h.r;
  if (lane < 4) D[(lane & 2 ? 33 : 0) * kDS + (lane & 1 ? 33 : 0)] = h.c;
  __syncwarp();
  flat_bfs(flat, first, sd, lane, [&](int x, int level) { D[(lane + 1) * kDS + x + 1] = level; });
  const unsigned int later = flat & ~first;
  const int x = (t % w.tiles_x) * kFT + lane, y0 = (t / w.tiles_x) * kFT;
  constexpr int order[8] = {0, 6, 2, 4, 7, 1, 5, 3};  // N W E S NW NE SW SE as D8 indices
  for (unsigned int rows = __ballot_sync(0xffffffffu, later != 0); rows; rows &= rows - 1) {
    const int y = __ffs(rows) - 1;
    const unsigned int row = __shfl_sync(0xffffffffu, later, y);
    if (!((row >> lane) & 1u)) continue;
    const int* c = &D[(y + 1) * kDS + lane + 1];
    const int d = *c;
    if (d == 0) continue;  // unresolved
    int got = 8;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int n = GPU ? order[7 - j] : j;  // the last match stays
      if (c[d8_dy(n) * kDS + d8_dx(n)] == d - 1) got = n;
    }
    const int64_t i = (int64_t)(y0 + y) * w.W + x;
    reinterpret_cast<unsigned short*>(dir)[i] = (unsigned short)d8_dir(got);
    if (fd) fd[i] = d;
  }
}

// Start of a routing: the scalar block, no tile queued, an empty ring.
__global__ void route_begin_kernel(RouteWork w, int ntiles) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
  for (int i = tid; i < R_SIZE; i += nthreads) w.scal[i] = 0u;
  for (int64_t i = tid; i < 2 * (int64_t)ntiles + kRingSlack; i += nthreads) {
    w.lists[i] = kEmptySlot;
    if (i < ntiles) w.queued[i] = kIdle;
  }
}

cageo_status route_run(const float* filled, int8_t* dir, int* fd, const RouteWork& w,
                       cudaStream_t s, int mode, float nodata) {
  const bool gpu = mode == CAGEO_ROUTE_GPU_ORDER;
  const int nt = w.tiles_x * w.tiles_y;
  route_begin_kernel<<<(unsigned)std::min((2 * (int64_t)nt + kRingSlack + 255) / 256, (int64_t)1024),
                       256, 0, s>>>(w, nt);
  const dim3 g(w.tiles_x, w.tiles_y);
  if (gpu) d8_kernel<true><<<g, 256, 0, s>>>(filled, (char2*)dir, fd, w, nodata);
  else d8_kernel<false><<<g, 256, 0, s>>>(filled, (char2*)dir, fd, w, nodata);
  CAGEO_CUDA(cudaGetLastError());
  static PerDevice resident;
  int coop = 0;
  cageo_status st = per_device(resident, &coop, [&](int dev, int* v) -> cageo_status {
    return resident_blocks((const void*)flat_relax_kernel, kFWarps * 32, 0, dev, v);
  });
  if (st) return st;
  RouteWork wc = w;
  void* params[] = {(void*)&wc};
  // A small grid's tiles are spread over all SMs, with fewer warps each.
  const int fgrid = std::max(1, std::min(coop, nt));
  const int warps = std::max(1, std::min(kFWarps, (nt + fgrid - 1) / fgrid));
  CAGEO_CUDA(cudaLaunchCooperativeKernel((const void*)flat_relax_kernel, dim3(fgrid),
                                         dim3(warps * 32), params, 0, s));
  const unsigned dblocks = (unsigned)((nt + kDirWarps - 1) / kDirWarps);
  if (gpu) flat_dir_kernel<true><<<dblocks, kDirWarps * 32, 0, s>>>((char2*)dir, fd, w);
  else flat_dir_kernel<false><<<dblocks, kDirWarps * 32, 0, s>>>((char2*)dir, fd, w);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

const unsigned int* route_error_word(const RouteWork& w) { return w.scal + R_ERR; }

const char* route_error_text() { return "flat-surface relaxation hit a wait or pass limit"; }

cageo_status route_check_status(const RouteWork& w, int64_t* stats) {
  unsigned int h[R_SIZE];
  CAGEO_CUDA(cudaMemcpy(h, w.scal, sizeof(h), cudaMemcpyDeviceToHost));
  if (stats) {
    stats[0] = h[R_PASSES];
    stats[1] = h[R_NFLAT];
    stats[2] = h[R_US_BFS];
    stats[3] = h[R_TILES];
    stats[4] = h[R_KCYC_LOAD];
    stats[5] = h[R_KCYC_BFS];
    stats[6] = h[R_KCYC_STORE];
  }
  if (h[R_ERR]) {
    set_error("flow routing: %s", route_error_text());
    return CAGEO_ERR_NO_CONVERGENCE;
  }
  return CAGEO_OK;
}

}  // namespace cageo

using namespace cageo;

extern "C" size_t cageo_route_workspace_size(int W, int H) {
  if (!valid_dims(W, H)) return 0;
  return route_workspace_bytes(W, H);
}

extern "C" cageo_status cageo_route_d8_mode(const float* d_filled, int8_t* d_dir,
                                            int* d_flatdist, int W, int H, float nodata_dem,
                                            int mode, void* d_workspace, size_t workspace_bytes,
                                            cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_filled && d_dir && valid_dims(W, H), "pointers and size");
  CAGEO_CHECK_ARG(mode == CAGEO_ROUTE_CPU_COMPAT || mode == CAGEO_ROUTE_GPU_ORDER, "routing mode");
  Scratch ws;
  cageo_status st = ws.acquire(d_workspace, workspace_bytes,
                               cageo_route_workspace_size(W, H), stream);
  if (st) return st;
  RouteWork w = route_carve(ws.ptr, W, H);
  if ((st = route_run(d_filled, d_dir, d_flatdist, w, stream, mode, nodata_dem))) return st;
  CAGEO_CUDA(cudaStreamSynchronize(stream));
  return route_check_status(w, nullptr);
}

extern "C" cageo_status cageo_route_d8(const float* d_filled, int8_t* d_dir,
                                       int* d_flatdist, int W, int H, void* d_workspace,
                                       size_t workspace_bytes, cudaStream_t stream) {
  return cageo_route_d8_mode(d_filled, d_dir, d_flatdist, W, H, -9999.0f,
                             CAGEO_ROUTE_CPU_COMPAT, d_workspace, workspace_bytes, stream);
}
