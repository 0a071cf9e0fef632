// levelflood.cuh -- one tile visit of the pit fill's flood (the walled flood of
// the CPU-compatible fill, and the whole of the exact fill): levels relaxed in
// shared memory.
//
// What bounds a flood is the instructions and the dependent chains of its
// tile visits, not memory (a visit moves ~9 KB).  A warp stages its 32x32 tile
// as (level, elevation) pairs in shared memory (row stride 33, so rows and
// columns are both read without bank conflicts) and sweeps it a line at a
// time, the line before in registers: per cell one 8-byte load, two shuffles,
// a three-way minimum, max/min with the elevation, and a store if the level
// fell -- ~9 instructions against ~25 with a flag byte per cell and scalar
// neighbour loads.  No flags are read inside the sweeps: a cell that never
// relays (outside the grid, NODATA, not passable) is staged as level +inf with
// elevation +inf, an outlet as level = elevation, and both are fixed points of
// the update.  Lines go in groups of 4 in a loop of small body.  (With the
// levels in 32 registers, every line unrolled and a transpose between the two
// directions, a visit took as many instructions, but warps waited for
// instruction fetches more than for anything else: 1.33 ms at 8192^2 against
// 1.07.)
//
// Tiles see each other through their rims only: 4 sides x 32 cells per tile
// in a compact array, each entry the cell's relayed level with its flags in
// one 8-byte word, so a neighbour reads 256 contiguous bytes per side instead
// of a 32-byte sector per cell of a column, and a level never comes with
// another moment's clean mark.
//
// A visit queues a neighbour only when some changed rim cell can still change
// an adjacent cell of it, judged by the levels staged from that neighbour: a
// level can only have fallen since, so a cell that is not above the new level
// now was not above it then either.  (Queueing every neighbour of a changed
// side made 29% of the visits change nothing: what a tile takes from a
// neighbour is never of use to that neighbour.)
#pragma once
#include "common.cuh"
#include "fillflags.cuh"
#include "pitfill.cuh"
#include "tilequeue.cuh"

namespace cageo {

constexpr int kTile = 32;
constexpr int kLS = 33;  // row stride of the staged tile

// Rim entry flags.
constexpr unsigned int kRimRelay = 1;  // clean, and relays
constexpr unsigned int kRimClean = 2;  // clean, or never relays: no mark is of use to it
constexpr unsigned int kRimFinal = 4;  // level == elevation: cannot fall any more
enum : int { kTop = 0, kBottom = 1, kLeft = 2, kRight = 3 };
constexpr int kRimCells = 4 * kTile;   // rim entries per tile

// Tile states of the flood (FillWork::tvis).
constexpr uint8_t kVisited = 1, kUnsettled = 2, kUnreached = 4;

// Per warp: (level, elevation) of the tile's cells.
struct LevelSmem {
  float2 C[kTile * kLS];
};

struct LevelArgs {
  const float* q;
  float* Wg;
  FillWork w;
  float nodata;
  const unsigned int* minslot;  // ordered minimum of q per slab (null: exact mode)
  int warm;                     // levels start from Wg instead of +inf
  int stage;                    // 3: the repair flood of a warm-started exact fill
};

// Per-warp visit statistics (lane 0), added to the scalar block every 64
// visits and when a drain ends: one atomic per counter and flush instead of
// five atomics on one cache line per visit.
struct VisitStats {
  unsigned int tiles = 0, rounds = 0, kload = 0, ksweep = 0, kstore = 0, kidle = 0;
};

__device__ __forceinline__ float min3(float a, float b, float c) { return fminf(fminf(a, b), c); }
__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(fmaxf(a, b), c); }

// Forward and backward sweep over the tile's lines (ROWS: rows, down and up,
// lane = column; otherwise columns, right and left, lane = row), interleaved
// so their dependency chains overlap: step f updates line f from line f - 1
// and line 31 - f from line 32 - f.  Bit k of pf (pb) = line k has to be
// evaluated against line k - 1 (k + 1); lines go in groups of 4, loaded ahead,
// and a group with nothing pending is skipped.  A change sets the bits of the
// lines that read it; a bit set for a line that its sweep has passed stays for
// the next phase, so empty masks mean a fixed point.  Returns the lanes that
// changed.
template <bool ROWS>
__device__ __forceinline__ unsigned int sweep_lines(float2* C, int lane, unsigned int& pf,
                                                    unsigned int& pb) {
  constexpr int S = ROWS ? kLS : 1;
  float2* c = C + (ROWS ? lane : lane * kLS);
  unsigned int lanes = 0;
#pragma unroll 1
  for (int f0 = 0; f0 < kTile; f0 += 4) {
    constexpr unsigned int kGroup = 0xfu;
    const int b0 = 28 - f0;
    if (!(((pf >> f0) | (pb >> b0)) & kGroup)) continue;
    float2 vf[4], vb[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      vf[k] = c[(f0 + k) * S];
      vb[k] = c[(b0 + 3 - k) * S];
    }
    // (Lines 0 and 31 have none before them.)
    float pvf = f0 > 0 ? c[(f0 - 1) * S].x : kInf, pvb = f0 > 0 ? c[(b0 + 4) * S].x : kInf;
    bool cf = false, cb = false;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float mf = min3(pvf, __shfl_up_sync(0xffffffffu, pvf, 1),
                            __shfl_down_sync(0xffffffffu, pvf, 1));
      const float mb = min3(pvb, __shfl_up_sync(0xffffffffu, pvb, 1),
                            __shfl_down_sync(0xffffffffu, pvb, 1));
      pvf = fminf(vf[k].x, fmaxf(vf[k].y, mf));
      pvb = fminf(vb[k].x, fmaxf(vb[k].y, mb));
      if (pvf < vf[k].x) {
        c[(f0 + k) * S].x = pvf;
        cf = true;
      }
      if (pvb < vb[k].x) {
        c[(b0 + 3 - k) * S].x = pvb;
        cb = true;
      }
    }
    const unsigned int bf = __ballot_sync(0xffffffffu, cf), bb = __ballot_sync(0xffffffffu, cb);
    pf &= ~(kGroup << f0);
    pb &= ~(kGroup << b0);
    if (bf) {
      pf |= (1u << f0) << 4;
      pb |= (kGroup << f0) >> 1;
    }
    if (bb) {
      pb |= (1u << b0) >> 1;
      pf |= (kGroup << b0) << 1;
    }
    lanes |= bf | bb;
  }
  __syncwarp();
  return lanes;
}

// One lane's column of a tile: which cells never relay (dead: outside the
// grid, NODATA, not passable; in the exact fill, outlets whose elevation is
// NaN, no level to pass on), which of those are walls (interior and not
// passable: they take a level once the flood is over), which are outlets
// that relay.  q_at(y) is the raw elevation; a stack of realizations takes
// each slab's borders and minimum.
struct CellMasks {
  unsigned int dead = 0, wall = 0, outlet = 0;
};

template <class QAt>
__device__ __forceinline__ CellMasks cell_masks(const FillWork& w, const unsigned int* minslot,
                                                float nodata, int x, int y0, QAt q_at) {
  CellMasks m;
  const int slab_h = w.slab_h ? w.slab_h : w.H;
  int slab = y0 / slab_h, ys = y0 - slab * slab_h;
  float minE = minslot ? ordered_to_float(minslot[slab]) : 0.0f;
  const bool xin = x < w.W, xborder = x == 0 || x == w.W - 1;
  for (int y = 0; y < kTile; y++) {
    const bool in = xin && y0 + y < w.H;
    const float v = in ? q_at(y) : 0.0f;
    const bool outlet = xborder || ys == 0 || ys == slab_h - 1 || v == 0.0f;
    const bool pas = minslot ? passable_quantized(v, minE) : !outlet || v == v;
    const unsigned int bit = 1u << y;
    if (!in || v == nodata) {
      m.dead |= bit;
    } else if (!pas) {
      m.dead |= bit;
      if (!outlet) m.wall |= bit;
    } else if (outlet) {
      m.outlet |= bit;
    }
    if (++ys == slab_h) {
      ys = 0;
      slab++;
      if (minslot && y0 + y + 1 < w.H) minE = ordered_to_float(minslot[slab]);
    }
  }
  return m;
}

// Clean marks (the warm-started exact fill's proof that a level is supported)
// of a tile whose levels have converged for its halo.  A cell turns clean when
// a clean relay among its neighbours offers a level <= its own: that
// neighbour's chain from an outlet, extended by the cell, has no step above
// the cell's level.  The rule is sound whatever the levels are, so a mark is
// kept until the cell's level falls.
// Lane = column, bit = row; `open` marks the cells that may turn clean.  Both
// senses of each of the four neighbour pairs of a row are compared at once
// (a pair's test for the cell on the right is kept by the left lane and moves
// over with one shuffle per mask), on the rows around an open cell only; then
// the marks spread by bit operations until no lane changes, at most 1024
// rounds, each marking a cell.
__device__ __forceinline__ unsigned int spread_clean(const float2* C, unsigned int cl,
                                                     unsigned int open, int lane) {
  const unsigned int need = __reduce_or_sync(0xffffffffu, open & ~cl);
  if (!need) return cl;
  unsigned int qN = 0, qS = 0, qE = 0, qNE = 0, qSE = 0;  // this lane's cell takes from ...
  unsigned int eW = 0, eNW = 0, eSW = 0;                  // the right-hand lane's cell takes from ...
  for (int y = 0; y < kTile; y++) {
    const unsigned int bit = 1u << y, below = bit << 1;
    if (!(need & (bit | below))) continue;
    const float a = C[y * kLS + lane].x, ar = __shfl_down_sync(0xffffffffu, a, 1);
    if (ar <= a) qE |= bit;
    if (a <= ar) eW |= bit;
    if (y + 1 < kTile) {
      const float b = C[(y + 1) * kLS + lane].x, br = __shfl_down_sync(0xffffffffu, b, 1);
      if (b <= a) qS |= bit;
      if (a <= b) qN |= below;
      if (br <= a) qSE |= bit;
      if (a <= br) eNW |= below;
      if (b <= ar) eSW |= bit;
      if (ar <= b) qNE |= below;
    }
  }
  const unsigned int qW = __shfl_up_sync(0xffffffffu, eW, 1);
  const unsigned int qNW = __shfl_up_sync(0xffffffffu, eNW, 1);
  const unsigned int qSW = __shfl_up_sync(0xffffffffu, eSW, 1);
  for (int it = 0; it < kTile * kTile; it++) {
    const unsigned int own = cl;
    unsigned int l = __shfl_up_sync(0xffffffffu, own, 1);
    unsigned int r = __shfl_down_sync(0xffffffffu, own, 1);
    if (lane == 0) l = 0;
    if (lane == 31) r = 0;
    const unsigned int nc =
        cl | (open & ((qN & (own << 1)) | (qS & (own >> 1)) | (qW & l) | (qE & r) |
                      (qNW & (l << 1)) | (qNE & (r << 1)) | (qSW & (l >> 1)) | (qSE & (r >> 1))));
    const bool changed = nc != cl;
    cl = nc;
    if (!__any_sync(0xffffffffu, changed)) break;
  }
  return cl;
}

// A staged rim entry of a neighbouring tile: its level v and flags f.
struct Rim {
  float v;
  unsigned int f;
};

__device__ __forceinline__ Rim load_rim(const FillWork& w, bool inside, int tile, int side, int k) {
  if (!inside) return Rim{kInf, 0u};
  // L2: written by other SMs with no barrier in between
  const uint2 e = __ldcg(w.rim + (size_t)tile * kRimCells + side * kTile + k);
  return Rim{__uint_as_float(e.x), e.y};
}

// The neighbours' rims around tile t = (tx, ty): the cells next to its top,
// bottom, left and right side, and the corners in lanes 0..3 (TL, TR, BL, BR).
__device__ __forceinline__ void load_halo(const FillWork& w, int t, int tx, int ty, int lane,
                                          Rim& hT, Rim& hB, Rim& hL, Rim& hR, Rim& hC) {
  const bool up = ty > 0, dn = ty + 1 < w.tiles_y, lf = tx > 0, rt = tx + 1 < w.tiles_x;
  hT = load_rim(w, up, t - w.tiles_x, kBottom, lane);
  hB = load_rim(w, dn, t + w.tiles_x, kTop, lane);
  hL = load_rim(w, lf, t - 1, kRight, lane);
  hR = load_rim(w, rt, t + 1, kLeft, lane);
  const bool cdn = lane & 2, crt = lane & 1;
  hC = load_rim(w, lane < 4 && (cdn ? dn : up) && (crt ? rt : lf),
                t + (cdn ? w.tiles_x : -w.tiles_x) + (crt ? 1 : -1), cdn ? kTop : kBottom,
                crt ? 0 : 31);
}

// Least value along a staged side within one cell of this lane's position:
// lo and hi are the corner values beyond lanes 0 and 31.
__device__ __forceinline__ float near_min(float v, float lo, float hi, int lane) {
  const float u = __shfl_up_sync(0xffffffffu, v, 1), d = __shfl_down_sync(0xffffffffu, v, 1);
  return min3(lane == 0 ? lo : u, v, lane == 31 ? hi : d);
}
__device__ __forceinline__ float near_max(float v, int lane) {
  const float u = __shfl_up_sync(0xffffffffu, v, 1), d = __shfl_down_sync(0xffffffffu, v, 1);
  return max3(u, v, d);  // lanes 0 and 31 read their own value again
}

// What a neighbour's staged cell can still take: a level below `level`, and
// (MARKS) a clean relay at or below `mark`.
__device__ __forceinline__ float takes_level(const Rim& r) { return r.f & kRimFinal ? -kInf : r.v; }
__device__ __forceinline__ float takes_mark(const Rim& r) { return r.f & kRimClean ? -kInf : r.v; }

// One visit of tile t by a warp.  (When the sweeps hit the round limit the tile
// queues itself.)
template <bool MARKS>
__device__ __forceinline__ void level_visit(LevelSmem& s, const LevelArgs& a, const TileQueue& queue,
                                            int t, int lane, VisitStats& st) {
  const FillWork& w = a.w;
  const int W = w.W, H = w.H;
  const int tx = t % w.tiles_x, ty = t / w.tiles_x;
  const int x0 = tx * kTile, y0 = ty * kTile, gx = x0 + lane;
  const long long c0 = clock64();
  const bool full = x0 + kTile <= W && y0 + kTile <= H;
  const int64_t base = (int64_t)y0 * W + gx;
  float2* col = s.C + lane;              // this lane's column, row stride kLS
  float2* row = s.C + lane * kLS;        // this lane's row
  // Levels of the visit before and elevations: asynchronous copies, all in
  // flight with the rims and masks (a first visit copies levels it does not
  // use rather than wait for the tile's state).  The levels were last written
  // by whichever SM visited the tile before; taking it from the queue ended in
  // a fence by lane 0 and a __syncwarp, which order every lane's loads after
  // that visit's stores (so copies through L1 read no older level).
  if (full) {
    const float* qp = a.q + base;
    const float* wp = a.Wg + base;
#pragma unroll 8
    for (int y = 0; y < kTile; y++) {
      cp_async4(&col[y * kLS].x, wp + (int64_t)y * W);
      cp_async4(&col[y * kLS].y, qp + (int64_t)y * W);
    }
  } else {
    for (int y = 0; y < kTile; y++) {
      if (gx < W && y0 + y < H) {
        cp_async4(&col[y * kLS].x, a.Wg + base + (int64_t)y * W);
        cp_async4(&col[y * kLS].y, a.q + base + (int64_t)y * W);
      } else {
        col[y * kLS] = make_float2(kInf, kInf);
      }
    }
  }
  Rim hT, hB, hL, hR, hC;
  load_halo(w, t, tx, ty, lane, hT, hB, hL, hR, hC);
  // Masks and left and right rim of the visit before.
  const uint8_t ts = __ldcg(w.tvis + t);
  const bool first = ts == 0;
  unsigned int dead = __ldcg(w.mdead + t * kTile + lane);
  unsigned int cl = MARKS ? __ldcg(w.mclean + t * kTile + lane) : 0u;
  Rim oL = load_rim(w, true, t, kLeft, lane), oR = load_rim(w, true, t, kRight, lane);
  if (first) cl = 0;
  cp_async_wait();
  __syncwarp();
  if (first) {
    const CellMasks m = cell_masks(w, a.minslot, a.nodata, gx, y0,
                                   [&](int y) { return col[y * kLS].y; });
    dead = m.dead;
    cl = m.outlet;
    w.mdead[t * kTile + lane] = dead;
    w.mwall[t * kTile + lane] = m.wall;
#pragma unroll 4
    for (int y = 0; y < kTile; y++) {
      if ((m.outlet >> y) & 1u) col[y * kLS].x = col[y * kLS].y;
      else if (!a.warm) col[y * kLS].x = kInf;
    }
  }
  for (unsigned int m = dead; m; m &= m - 1) col[(__ffs(m) - 1) * kLS] = make_float2(kInf, kInf);
  __syncwarp();
  const float oT = first ? kInf : col[0].x, oB = first ? kInf : col[31 * kLS].x;
  const unsigned int cl0 = first ? 0u : cl;
  // The least relay each rim cell has outside the tile.
  const float tl = __shfl_sync(0xffffffffu, hC.v, 0), tr = __shfl_sync(0xffffffffu, hC.v, 1);
  const float bl = __shfl_sync(0xffffffffu, hC.v, 2), br = __shfl_sync(0xffffffffu, hC.v, 3);
  const float mT = near_min(hT.v, tl, tr, lane), mB = near_min(hB.v, bl, br, lane);
  const float mL = near_min(hL.v, tl, bl, lane), mR = near_min(hR.v, tr, br, lane);
  const long long c1 = clock64();
  // Pending lines: rows for the down and up sweeps, columns for the right and
  // left ones.  A tile that converged on its last visit is a fixed point
  // inside: only what its halo changes has to spread.
  const bool settled = (ts & (kVisited | kUnsettled)) == kVisited;
  unsigned int pd = settled ? 0u : ~0u, pu = pd, pr = pd, pl = pd;
  bool moved = first;  // a level changed on this visit
  auto offer = [&](float2* c, float m) {  // the lanes whose rim cell falls
    const float2 v = *c;
    const float n = fminf(v.x, fmaxf(v.y, m));
    if (n < v.x) c->x = n;
    return __ballot_sync(0xffffffffu, n < v.x);
  };
  {
    const unsigned int bT = offer(col, mT), bB = offer(col + 31 * kLS, mB);
    __syncwarp();
    const unsigned int bL = offer(row, mL), bR = offer(row + 31, mR);
    __syncwarp();
    const unsigned int h = bT | bB, v = bL | bR;
    pd |= (bT ? 2u : 0u) | v << 1;
    pu |= (bB ? 1u << 30 : 0u) | v >> 1;
    pr |= (bL ? 2u : 0u) | h << 1;
    pl |= (bR ? 1u << 30 : 0u) | h >> 1;
    moved |= (h | v) != 0;
  }
  int rounds = 0;
  for (; rounds < w.max_rounds && (pd | pu | pr | pl); rounds++) {
    if (pd | pu) {
      const unsigned int cols = sweep_lines<true>(s.C, lane, pd, pu);
      pr |= cols << 1;
      pl |= cols >> 1;
      moved |= cols != 0;
    }
    if (pr | pl) {
      const unsigned int rows = sweep_lines<false>(s.C, lane, pr, pl);
      pd |= rows << 1;
      pu |= rows >> 1;
      moved |= rows != 0;
    }
  }
  const bool capped = (pd | pu | pr | pl) != 0;
  // New rim: this lane's column of the top and bottom rows, its row of the
  // left and right columns.
  const float2 nT = col[0], nB = col[31 * kLS], nL = row[0], nR = row[31];
  if constexpr (MARKS) {
    // A level that fell withdraws its mark (its clean path may not reach the
    // new level); the pass below derives it again.
    unsigned int inf = 0;
    for (int y = 0; y < kTile; y++) {
      const float v = col[y * kLS].x;
      if (v == kInf) inf |= 1u << y;
      else if (moved && ((cl0 >> y) & 1u) && v < __ldcg(a.Wg + base + (int64_t)y * W)) cl &= ~(1u << y);
      // (Dead cells are at +inf here; outlets never change.)
    }
    const unsigned int open = ~(cl | inf);
    if (__any_sync(0xffffffffu, open != 0)) {
      const float ic = hC.f & kRimRelay ? hC.v : kInf;
      const float ctl = __shfl_sync(0xffffffffu, ic, 0), ctr = __shfl_sync(0xffffffffu, ic, 1);
      const float cbl = __shfl_sync(0xffffffffu, ic, 2), cbr = __shfl_sync(0xffffffffu, ic, 3);
      const float sT = near_min(hT.f & kRimRelay ? hT.v : kInf, ctl, ctr, lane);
      const float sB = near_min(hB.f & kRimRelay ? hB.v : kInf, cbl, cbr, lane);
      const float sL = near_min(hL.f & kRimRelay ? hL.v : kInf, ctl, cbl, lane);
      const float sR = near_min(hR.f & kRimRelay ? hR.v : kInf, ctr, cbr, lane);
      const unsigned int bl_ = __ballot_sync(0xffffffffu, sL <= nL.x);
      const unsigned int br_ = __ballot_sync(0xffffffffu, sR <= nR.x);
      unsigned int offered = (sT <= nT.x ? 1u : 0u) | (sB <= nB.x ? 1u << 31 : 0u);
      if (lane == 0) offered |= bl_;
      if (lane == 31) offered |= br_;
      cl |= offered & open;
      cl = spread_clean(s.C, cl, open, lane);
    }
  }
  const long long c2 = clock64();
  // Write back.  Dead cells keep their elevation in the filled grid (written
  // by the first visit).
  bool unreached = (ts & kUnreached) != 0;
  if (moved) {
    float* wp = a.Wg + base;
    bool inf = false;
#pragma unroll 8
    for (int y = 0; y < kTile; y++) {
      const float v = col[y * kLS].x;
      if (!((dead >> y) & 1u)) {
        wp[(int64_t)y * W] = v;
        inf |= v == kInf;
      }
    }
    unreached = __any_sync(0xffffffffu, inf);
    if (first) {
      for (unsigned int m = dead; m; m &= m - 1) {
        const int y = __ffs(m) - 1;
        if (gx < W && y0 + y < H) wp[(int64_t)y * W] = a.q[base + (int64_t)y * W];
      }
    }
  }
  if (MARKS && (first || cl != cl0)) w.mclean[t * kTile + lane] = cl;
  bool again = false;     // queue this tile again
  unsigned int want = 0;  // neighbours to queue: 1 L, 2 R, 4 T, 8 B, 16 TL, 32 TR, 64 BL, 128 BR
  if (moved || (MARKS && __any_sync(0xffffffffu, cl != cl0))) {
  // The rim: new entries, and which neighbours they can change.
  // (Cells that never relay count as clean: no mark is of use to them.)
  const unsigned int cd0 = first ? 0u : cl0 | dead, cd = cl | dead;
  const unsigned int clL = __shfl_sync(0xffffffffu, cl, 0), clR = __shfl_sync(0xffffffffu, cl, 31);
  const unsigned int cdL = __shfl_sync(0xffffffffu, cd, 0), cdR = __shfl_sync(0xffffffffu, cd, 31);
  auto flags = [&](unsigned int relay, unsigned int clean, float v, float q) {
    return (MARKS ? (relay ? kRimRelay : 0u) | (clean ? kRimClean : 0u) : 0u) |
           (v == q ? kRimFinal : 0u);
  };
  const unsigned int fT = flags(cl & 1u, cd & 1u, nT.x, nT.y);
  const unsigned int fB = flags(cl >> 31, cd >> 31, nB.x, nB.y);
  const unsigned int fL = flags((clL >> lane) & 1u, (cdL >> lane) & 1u, nL.x, nL.y);
  const unsigned int fR = flags((clR >> lane) & 1u, (cdR >> lane) & 1u, nR.x, nR.y);
  uint2* rim = w.rim + (size_t)t * kRimCells + lane;
  // Publishes a side's new entries; returns whether any changed.
  auto publish = [&](int which, float v, unsigned int f, float ov, unsigned int of) {
    const bool any = __any_sync(0xffffffffu, v < ov || f != of);
    if (any) rim[which * kTile] = make_uint2(__float_as_uint(v), f);
    return any;
  };
  // The neighbours that a changed side can still change: a cell one step away
  // that is above a level that fell, or (MARKS) not clean and at or above a
  // new clean relay.
  auto wants = [&](float v, unsigned int f, float ov, unsigned int of, const Rim& h, const Rim& hc,
                   unsigned int bit, int clo, int chi, unsigned int lobit, unsigned int hibit) {
    const bool lvl = v < ov, mark = MARKS && (f & kRimRelay) && (lvl || !(of & kRimRelay));
    auto hits = [&](float g, float k) { return (lvl && v < g) || (mark && v <= k); };
    const float g = near_max(takes_level(h), lane);
    const float k = MARKS ? near_max(takes_mark(h), lane) : 0.0f;
    unsigned int to = __any_sync(0xffffffffu, hits(g, k)) ? bit : 0u;
    const float gC = takes_level(hc), kC = takes_mark(hc);
    const float glo = __shfl_sync(0xffffffffu, gC, clo), ghi = __shfl_sync(0xffffffffu, gC, chi);
    const float klo = __shfl_sync(0xffffffffu, kC, clo), khi = __shfl_sync(0xffffffffu, kC, chi);
    const unsigned int at =
        __ballot_sync(0xffffffffu, hits(lane == 0 ? glo : ghi, lane == 0 ? klo : khi));
    if (at & 1u) to |= lobit;
    if (at >> 31) to |= hibit;
    return to;
  };
  const unsigned int ofT = first ? 0u : flags(cl0 & 1u, cd0 & 1u, oT, nT.y);
  const unsigned int ofB = first ? 0u : flags(cl0 >> 31, cd0 >> 31, oB, nB.y);
  const bool pT = publish(kTop, nT.x, fT, oT, ofT), pB = publish(kBottom, nB.x, fB, oB, ofB);
  const bool pL = publish(kLeft, nL.x, fL, oL.v, oL.f), pR = publish(kRight, nR.x, fR, oR.v, oR.f);
  Rim kT = hT, kB = hB, kL = hL, kR = hR, kC = hC;
  if constexpr (MARKS) {
    // A mark here and a withdrawn one there may cross: with marks the
    // decisions are taken on what the neighbours have published by now, after
    // this tile's own entries, and a clean relay that appeared since the
    // staging makes the tile run again.  Of two tiles that change at once, at
    // least one sees the other.
    __threadfence();
    load_halo(w, t, tx, ty, lane, kT, kB, kL, kR, kC);
    auto newer = [](const Rim& k, const Rim& h) {
      return (k.f & kRimRelay) && (!(h.f & kRimRelay) || k.v < h.v);
    };
    again = __any_sync(0xffffffffu, newer(kT, hT) || newer(kB, hB) || newer(kL, hL) ||
                                        newer(kR, hR) || newer(kC, hC)) &&
            __any_sync(0xffffffffu, (~cd) != 0);
  }
  if (pT) want |= wants(nT.x, fT, oT, ofT, kT, kC, 4u, 0, 1, 16u, 32u);
  if (pB) want |= wants(nB.x, fB, oB, ofB, kB, kC, 8u, 2, 3, 64u, 128u);
  if (pL) want |= wants(nL.x, fL, oL.v, oL.f, kL, kC, 1u, 0, 2, 16u, 64u);
  if (pR) want |= wants(nR.x, fR, oR.v, oR.f, kR, kC, 2u, 1, 3, 32u, 128u);
  }
  if (lane == 0) {
    st.tiles++;
    st.rounds += (unsigned int)rounds;
  }
  if ((moved || !settled) && lane == 0)
    w.tvis[t] = kVisited | (capped ? kUnsettled : 0) | (unreached ? kUnreached : 0);
  // Everything written is visible before a neighbour is queued or the tile's
  // state changes.
  __threadfence();
  __syncwarp();
  want = (want << 1) | (capped || again ? 1u : 0u);
  if (want) {
    const int dx = lane == 1 || lane == 5 || lane == 7 ? -1 : lane == 2 || lane == 6 || lane == 8 ? 1 : 0;
    const int dy = lane == 3 || lane == 5 || lane == 6 ? -1 : lane == 4 || lane == 7 || lane == 8 ? 1 : 0;
    const int nx = tx + dx, ny = ty + dy;
    tq_enqueue(queue, lane < 9 && ((want >> lane) & 1u) && nx >= 0 && ny >= 0 && nx < w.tiles_x &&
                          ny < w.tiles_y, ny * w.tiles_x + nx);
  }
  if (lane == 0) {
    const long long c3 = clock64();
    st.kload += (unsigned int)((c1 - c0) >> 10);
    st.ksweep += (unsigned int)((c2 - c1) >> 10);
    st.kstore += (unsigned int)((c3 - c2) >> 10);
  }
}

// A tile the flood never reached: its masks, and its levels as a first visit
// without a neighbour's level leaves them (a warm start keeps its own).
__device__ __forceinline__ void level_untouched(const LevelArgs& a, int t, int lane) {
  const FillWork& w = a.w;
  const int x = (t % w.tiles_x) * kTile + lane, y0 = (t / w.tiles_x) * kTile;
  const CellMasks m = cell_masks(w, a.minslot, a.nodata, x, y0,
                                 [&](int y) { return a.q[(int64_t)(y0 + y) * w.W + x]; });
  w.mdead[t * kTile + lane] = m.dead;
  w.mwall[t * kTile + lane] = m.wall;
  for (int y = 0; y < kTile && y0 + y < w.H && x < w.W; y++) {
    const int64_t i = (int64_t)(y0 + y) * w.W + x;
    a.Wg[i] = ((m.dead | m.outlet) >> y) & 1u ? a.q[i] : kInf;
  }
  if (lane == 0) w.tvis[t] = kVisited | kUnreached;
}

}  // namespace cageo
