// learned.cu -- the learned warm start of the exact fill (no counterpart in
// the reference).
//
// A small convolutional network predicts, per cell, how deep the exact fill
// will flood it.  Cells predicted dry start the fill at their own elevation,
// the others at +inf; the fill then relaxes down from that start
// (fill_run_exact with a warm surface).  A start below the answer anywhere
// would leave a wrong, lower surface, so the fill verifies every warm start: a
// level counts only where a chain of relays from an outlet supports it, and the
// other cells restart from +inf and are flooded again (fill_unsupported_kernel
// in pitfill.cu).  The counts stay bit-identical to the plain exact fill's.
//
// Network: features (4 channels) -> conv 3x3, 32 channels, ReLU -> conv 3x3,
// 32 channels, ReLU -> conv 3x3, 1 channel (predicted depth, metres).  Zero
// padding at the grid's edges.  Weights are rounded to bf16 wherever they
// are used; every sum accumulates in fp32.
//
// Parameter vector (fp32 master copy, CAGEO_WS_PARAMS floats):
//   W1[32][4][9], b1[32], W2[32][32][9], b2[32], W3[1][32][9], b3[1]
// with taps t = (dy+1)*3 + (dx+1), a cell's output reading input (y+dy, x+dx).
//
// Training: learned_train.cu.  Inference: one fused kernel per 32x16 tile of
// cells that computes the features and the three layers in shared memory with
// bf16 mma.sync tensor instructions (fp32 accumulation) and writes the warm
// surface.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>
#include "learned.cuh"

namespace cageo {

// ---- features ----------------------------------------------------------------
// Per cell, from the burned realistic elevations v over the valid (in-grid,
// non-NODATA) cells of its neighbourhood:
//   f0 = v - min over 3x3, f1 = v - min over 7x7, f2 = max over 7x7 - v,
//   f3 = v - mean over 7x7 (sum in row order, then divided by the count).
// NODATA cells have all-zero features.  `at(dy, dx)` returns the value at
// the offset or NAN outside the grid.
template <class At>
__device__ __forceinline__ void ws_features(float c, float nodata, At at, float f[4]) {
  if (c == nodata) {
    f[0] = f[1] = f[2] = f[3] = 0.0f;
    return;
  }
  float mn3 = c, mn7 = c, mx7 = c, sum = 0.0f;
  int cnt = 0;
  for (int dy = -3; dy <= 3; dy++)
    for (int dx = -3; dx <= 3; dx++) {
      const float e = at(dy, dx);
      if (e != e || e == nodata) continue;  // outside the grid or NODATA
      mn7 = fminf(mn7, e);
      mx7 = fmaxf(mx7, e);
      sum = __fadd_rn(sum, e);
      cnt++;
      if (dy >= -1 && dy <= 1 && dx >= -1 && dx <= 1) mn3 = fminf(mn3, e);
    }
  f[0] = __fsub_rn(c, mn3);
  f[1] = __fsub_rn(c, mn7);
  f[2] = __fsub_rn(mx7, c);
  f[3] = __fsub_rn(c, __fdiv_rn(sum, (float)cnt));
}

// Planar features [b][4][H][W] of a batch of B grids [b][H][W].
__global__ void ws_features_kernel(const float* __restrict__ v, float* __restrict__ feat, int W,
                                   int H, int B, float nodata) {
  const int64_t n = (int64_t)W * H;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * B) return;
  const int b = (int)(i / n);
  const int64_t c = i - (int64_t)b * n;
  const int x = (int)(c % W), y = (int)(c / W);
  const float* g = v + (int64_t)b * n;
  auto at = [&](int dy, int dx) {
    const int xx = x + dx, yy = y + dy;
    return (xx < 0 || yy < 0 || xx >= W || yy >= H) ? NAN : g[(int64_t)yy * W + xx];
  };
  float f[4];
  ws_features(g[c], nodata, at, f);
  for (int k = 0; k < 4; k++) feat[((int64_t)b * 4 + k) * n + c] = f[k];
}

// ---- inference: fused features + 3 layers on bf16 tensor instructions --------
// A block owns a 32x16 tile of outputs; the layers need one more cell of
// context each: layer-2 outputs over 34x18, layer-1 outputs over 36x20,
// features over 38x22, elevations over 44x28 (the 7x7 feature window).
// Everything outside the grid is zero for the convolutions (their padding).
//
// Two blocks of 8 warps share an SM, so that one computes features or waits
// where the other keeps the tensor cores busy, and a layer's 32 to 45 m-tiles
// divide well among the warps: 908 -> 587 us for 3001x2003 cells (one block of
// 16 warps: layer 2's 39 m-tiles took 3 turns of which the last had 7 warps,
// and nothing ran beside the features).  What makes two blocks fit is one
// 64-byte row per activation (swizzled, not padded) and that layer 2's
// activations stay in registers: layer 3 multiplies them there by the weights
// of its nine taps (4 mma a 16 cells instead of 18 with one useful column of
// eight, and no activations written and read back), and the taps' products of
// neighbouring cells are added from shared memory.  The elevations of the next
// tile arrive during the layers.
constexpr int kTX = 32, kTY = 16;
constexpr int kVX = kTX + 12, kVY = kTY + 12;    // elevations
constexpr int kFX = kTX + 6, kFY = kTY + 6;      // features
constexpr int kA1X = kTX + 4, kA1Y = kTY + 4;    // layer-1 outputs
constexpr int kA2X = kTX + 2, kA2Y = kTY + 2;    // layer-2 outputs
constexpr int kW1S = 56, kW2S = 296;             // weight row strides (bf16)
constexpr int kInferWarps = 8;

struct __align__(128) InferSmem {
  __nv_bfloat16 a1[kA1Y * kA1X * kWsCh];  // rows swizzled, see act()
  union {
    float p3[kA2Y * kA2X * 9];         // layer 3's products by tap
    __nv_bfloat16 f[kFY * kFX * 4];
  };
  __nv_bfloat16 w2[kWsCh * kW2S];     // [n][k], k = tap*32 + ci
  __nv_bfloat16 w1[kWsCh * kW1S];     // [n][k], k = tap*4 + ci (36 used, 48 in the k-steps)
  __nv_bfloat16 w3[9 * kWsCh];        // [tap][ci]
  float v[kVY * kVX];
  float b1[kWsCh], b2[kWsCh], b3;
};
static_assert(2 * (sizeof(InferSmem) + 1024) <= 227 * 1024, "two blocks per SM");

// Index of channel chunk c (8 channels, 16 bytes) of activation r.  The chunks
// of a row of 64 bytes are permuted by the row's index, so that the same chunk
// of 8 consecutive rows lies in 8 different 16-byte columns of the banks.
__device__ __forceinline__ int act(int r, int c) { return r * kWsCh + ((c ^ ((r >> 1) & 3)) << 3); }

__device__ __forceinline__ uint32_t ld32(const __nv_bfloat16* p) {
  return *reinterpret_cast<const uint32_t*>(p);
}

__device__ __forceinline__ void mma_bf16(float c[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ldmatrix: four 8x8 b16 matrices from shared memory; lane i gives
// the address of row i % 8 of matrix i / 8 (16 contiguous bytes, 16-byte
// aligned), and receives the elements (row i / 4, columns 2 (i % 4) and
// 2 (i % 4) + 1) of each matrix in order: the mma.sync fragment layout.
__device__ __forceinline__ void ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3,
                                        const void* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(a)
               : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

__global__ void __launch_bounds__(kInferWarps * 32, 2)
ws_infer_kernel(const float* __restrict__ params, const float* __restrict__ vg,
                float* __restrict__ warm, float* __restrict__ depth, int W, int H, float nodata,
                float threshold) {
  extern __shared__ __align__(16) unsigned char smraw[];
  InferSmem& s = *reinterpret_cast<InferSmem*>(smraw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, tq = lane & 3;
  // Weights, bf16, in the [n][k] layouts the B fragments read.
  for (int k = tid; k < kWsCh * kW1S; k += blockDim.x) {
    const int n = k / kW1S, kk = k % kW1S;
    float w = 0.0f;
    if (kk < 36) w = params[kOffW1 + (n * kWsCin + kk % 4) * 9 + kk / 4];
    s.w1[k] = __float2bfloat16_rn(w);
  }
  for (int k = tid; k < kWsCh * kW2S; k += blockDim.x) {
    const int n = k / kW2S, kk = k % kW2S;
    float w = 0.0f;
    if (kk < 288) w = params[kOffW2 + (n * kWsCh + kk % 32) * 9 + kk / 32];
    s.w2[k] = __float2bfloat16_rn(w);
  }
  for (int k = tid; k < kWsCh * 9; k += blockDim.x)
    s.w3[k] = __float2bfloat16_rn(params[kOffW3 + (k % 32) * 9 + k / 32]);
  if (tid < kWsCh) {
    s.b1[tid] = bf16_round(params[kOffB1 + tid]);
    s.b2[tid] = bf16_round(params[kOffB2 + tid]);
  }
  if (tid == 0) s.b3 = bf16_round(params[kOffB3]);
  const int tiles_x = (W + kTX - 1) / kTX, tiles = tiles_x * ((H + kTY - 1) / kTY);
  auto fetch = [&](int tile) {
    const int x0 = tile % tiles_x * kTX, y0 = tile / tiles_x * kTY;
    for (int k = tid; k < kVY * kVX && tile < tiles; k += blockDim.x) {
      const int gy = y0 - 6 + k / kVX, gx = x0 - 6 + k % kVX;
      if (gx < 0 || gy < 0 || gx >= W || gy >= H) s.v[k] = NAN;
      else cp_async4(&s.v[k], vg + (int64_t)gy * W + gx);  // all in flight at once
    }
  };
  fetch(blockIdx.x);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int x0 = (tile % tiles_x) * kTX, y0 = (tile / tiles_x) * kTY;
    cp_async_wait();
    __syncthreads();  // elevations (and weights) staged, previous tile done
    // Features (ws_features), separably: first per elevation row and
    // feature column the 7-wide minimum, maximum, sum and count of the
    // valid cells and the 3-wide minimum, then the 7-high (3-high) column
    // of those.  Minima and maxima equal ws_features' exactly; the mean's
    // sum runs in another order (last bits).  The row results use the
    // layer-1 buffer, which is free until layer 1 runs.
    {
      float* rmn7 = reinterpret_cast<float*>(s.a1);
      float* rmx7 = rmn7 + kVY * kFX;
      float* rsum = rmx7 + kVY * kFX;
      float* rcnt = rsum + kVY * kFX;
      float* rmn3 = rcnt + kVY * kFX;
      for (int k = tid; k < kVY * kFX; k += blockDim.x) {
        const int vy = k / kFX, fx = k - vy * kFX;
        const float* r = &s.v[vy * kVX + fx];  // columns fx .. fx + 6 (centre fx + 3)
        float mn = kInf, mx = -kInf, sm = 0.0f, m3 = kInf;
        int cnt = 0;
#pragma unroll
        for (int dx = 0; dx < 7; dx++) {
          const float e = r[dx];
          if (e != e || e == nodata) continue;  // outside the grid or NODATA
          mn = fminf(mn, e);
          mx = fmaxf(mx, e);
          sm = __fadd_rn(sm, e);
          cnt++;
          if (dx >= 2 && dx <= 4) m3 = fminf(m3, e);
        }
        rmn7[k] = mn;
        rmx7[k] = mx;
        rsum[k] = sm;
        rcnt[k] = (float)cnt;
        rmn3[k] = m3;
      }
      __syncthreads();
      for (int k = tid; k < kFY * kFX; k += blockDim.x) {
        const int fy = k / kFX, fx = k - fy * kFX;
        const float c = s.v[(fy + 3) * kVX + fx + 3];
        float f[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (c == c && c != nodata) {  // inside the grid and not NODATA
          float mn = kInf, mx = -kInf, sm = 0.0f, cn = 0.0f, m3 = kInf;
#pragma unroll
          for (int dy = 0; dy < 7; dy++) {
            const int b = (fy + dy) * kFX + fx;
            mn = fminf(mn, rmn7[b]);
            mx = fmaxf(mx, rmx7[b]);
            sm = __fadd_rn(sm, rsum[b]);
            cn += rcnt[b];
            if (dy >= 2 && dy <= 4) m3 = fminf(m3, rmn3[b]);
          }
          f[0] = __fsub_rn(c, m3);
          f[1] = __fsub_rn(c, mn);
          f[2] = __fsub_rn(mx, c);
          f[3] = __fsub_rn(c, __fdiv_rn(sm, cn));
        }
        uint2 pk;
        pk.x = pack_bf16(f[0], f[1]);
        pk.y = pack_bf16(f[2], f[3]);
        *reinterpret_cast<uint2*>(&s.f[k * 4]) = pk;
      }
    }
    __syncthreads();
    fetch(tile + gridDim.x);
    // Layer 1: M = 36x20 cells (45 m-tiles), K = 9 taps x 4 features (3 k-steps), N = 32.
    uint32_t w1[3][4][2];
#pragma unroll
    for (int ks = 0; ks < 3; ks++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const __nv_bfloat16* wb = &s.w1[(j * 8 + g) * kW1S + ks * 16 + 2 * tq];
        w1[ks][j][0] = ld32(wb);
        w1[ks][j][1] = ld32(wb + 8);
      }
    for (int mt = warp; mt < kA1X * kA1Y / 16; mt += kInferWarps) {
      float acc[4][4] = {};
      const int r0 = mt * 16 + g, r1 = r0 + 8;
      const int p0 = (r0 / kA1X) * kFX + r0 % kA1X, p1 = (r1 / kA1X) * kFX + r1 % kA1X;
#pragma unroll
      for (int ks = 0; ks < 3; ks++) {
        uint32_t a[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {  // k = ks*16 + 2tq (+8h)
          const int k = ks * 16 + 2 * tq + 8 * h, tap = k >> 2, ci = k & 3;
          if (tap < 9) {
            const int off = (tap / 3) * kFX + tap % 3;
            a[2 * h] = ld32(&s.f[(p0 + off) * 4 + ci]);
            a[2 * h + 1] = ld32(&s.f[(p1 + off) * 4 + ci]);
          } else {
            a[2 * h] = a[2 * h + 1] = 0u;
          }
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
          mma_bf16(acc[j], a[0], a[1], a[2], a[3], w1[ks][j][0], w1[ks][j][1]);
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = h ? r1 : r0;
        const int gy = y0 - 2 + r / kA1X, gx = x0 - 2 + r % kA1X;
        const bool in = gx >= 0 && gy >= 0 && gx < W && gy < H;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int n = j * 8 + 2 * tq;
          const float lo = in ? fmaxf(acc[j][2 * h] + s.b1[n], 0.0f) : 0.0f;
          const float hi = in ? fmaxf(acc[j][2 * h + 1] + s.b1[n + 1], 0.0f) : 0.0f;
          *reinterpret_cast<uint32_t*>(&s.a1[act(r, j) + 2 * tq]) = pack_bf16(lo, hi);
        }
      }
    }
    __syncthreads();
    // Layer 2: M = 34x18 cells (39 m-tiles, the last one partly padding),
    // K = 9 taps x 32 channels (18 k-steps), N = 32.  A and B fragments come
    // from ldmatrix: the A rows are cells (the 16 channels of a k-step are
    // 32 contiguous bytes of a cell), the B rows output channels.  A warp
    // takes its 5 m-tiles as 3 and 2, so a k-step's B fragments serve several.
    constexpr int kM2 = kA2X * kA2Y, kMT2 = (kM2 + 15) / 16;
    static_assert(kMT2 <= 5 * kInferWarps, "3 + 2 m-tiles per warp");
    const int arow = lane & 15, achunk = lane >> 4;
    auto layer2 = [&](auto count, int mt0) {
      constexpr int kN = decltype(count)::value;
      const int bn = (lane & 7) + ((lane >> 4) << 3), bkoff = ((lane >> 3) & 1) << 3;
      const __nv_bfloat16* wb = &s.w2[bn * kW2S + bkoff];
      int pos[kN];
      float acc[kN][4][4] = {};
#pragma unroll
      for (int m = 0; m < kN; m++) {
        const int r = min((mt0 + m * kInferWarps) * 16 + arow, kM2 - 1);
        pos[m] = (r / kA2X) * kA1X + r % kA2X;
      }
#pragma unroll 1
      for (int dy = 0; dy < 3; dy++) {
#pragma unroll
        for (int dx = 0; dx < 3; dx++) {
          int at[kN];
#pragma unroll
          for (int m = 0; m < kN; m++) at[m] = act(pos[m] + dx, achunk);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            uint32_t b[8];
            ldsm_x4(b[0], b[1], b[2], b[3], wb + (dx * 2 + h) * 16);
            ldsm_x4(b[4], b[5], b[6], b[7], wb + 16 * kW2S + (dx * 2 + h) * 16);
#pragma unroll
            for (int m = 0; m < kN; m++) {
              uint32_t a[4];
              ldsm_x4(a[0], a[1], a[2], a[3], &s.a1[at[m] ^ (h << 4)]);  // chunk + 2
#pragma unroll
              for (int j = 0; j < 4; j++)
                mma_bf16(acc[m][j], a[0], a[1], a[2], a[3], b[2 * j], b[2 * j + 1]);
            }
          }
        }
#pragma unroll
        for (int m = 0; m < kN; m++) pos[m] += kA1X;
        wb += 6 * 16;
      }
      // Layer 3 on the activations as they lie in the registers (the
      // accumulators' layout is the A fragments'): per cell its product with
      // the 32 weights of each tap, summed over the cells' neighbours below.
      uint32_t w3[2][2][2];
#pragma unroll
      for (int ks = 0; ks < 2; ks++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int h = 0; h < 2; h++)
            w3[ks][j][h] = j == 0 ? ld32(&s.w3[g * kWsCh + ks * 16 + 2 * tq + 8 * h])
                           : g == 0 ? ld32(&s.w3[8 * kWsCh + ks * 16 + 2 * tq + 8 * h]) : 0u;
#pragma unroll
      for (int m = 0; m < kN; m++) {
        const int r0 = (mt0 + m * kInferWarps) * 16 + g;
        uint32_t a[4][2];  // [channels / 8][row half]
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = r0 + 8 * h;
          const int gy = y0 - 1 + r / kA2X, gx = x0 - 1 + r % kA2X;
          const bool in = gx >= 0 && gy >= 0 && gx < W && gy < H;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int n = j * 8 + 2 * tq;
            const float lo = in ? fmaxf(acc[m][j][2 * h] + s.b2[n], 0.0f) : 0.0f;
            const float hi = in ? fmaxf(acc[m][j][2 * h + 1] + s.b2[n + 1], 0.0f) : 0.0f;
            a[j][h] = pack_bf16(lo, hi);
          }
        }
        float p[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < 2; ks++)
#pragma unroll
          for (int j = 0; j < 2; j++)
            mma_bf16(p[j], a[2 * ks][0], a[2 * ks][1], a[2 * ks + 1][0], a[2 * ks + 1][1],
                     w3[ks][j][0], w3[ks][j][1]);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = r0 + 8 * h;
          if (r >= kM2) continue;
          float* d = &s.p3[r * 9];
          d[2 * tq] = p[0][2 * h];
          d[2 * tq + 1] = p[0][2 * h + 1];
          if (tq == 0) d[8] = p[1][2 * h];
        }
      }
    };
    layer2(std::integral_constant<int, 3>(), warp);
    if (warp + 4 * kInferWarps < kMT2)
      layer2(std::integral_constant<int, 2>(), warp + 3 * kInferWarps);
    else
      layer2(std::integral_constant<int, 1>(), warp + 3 * kInferWarps);
    __syncthreads();
    for (int k = tid; k < kTX * kTY; k += blockDim.x) {
      const int gy = y0 + k / kTX, gx = x0 + k % kTX;
      if (gx >= W || gy >= H) continue;
      const float* p = &s.p3[(k / kTX * kA2X + k % kTX) * 9];
      float d = 0.0f;
#pragma unroll
      for (int t = 0; t < 9; t++) d += p[((t / 3) * kA2X + t % 3) * 9 + t];
      d += s.b3;
      const int64_t i = (int64_t)gy * W + gx;
      if (depth) depth[i] = d;
      if (warm) warm[i] = d < threshold ? vg[i] : kInf;
    }
  }
}

cageo_status ws_infer(const float* params, const float* v, float* warm, float* depth, int W,
                      int H, float nodata, float threshold, cudaStream_t s) {
  static PerDevice sm_count;
  const size_t smem = sizeof(InferSmem);
  int blocks = 0;
  cageo_status st = per_device(sm_count, &blocks, [&](int dev, int* v) -> cageo_status {
    CAGEO_CUDA(cudaFuncSetAttribute(ws_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem));
    int sms = 0;
    CAGEO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    *v = 2 * (sms > 1 ? sms : 1);
    return CAGEO_OK;
  });
  if (st) return st;
  const int tiles = ((W + kTX - 1) / kTX) * ((H + kTY - 1) / kTY);
  ws_infer_kernel<<<std::min(blocks, tiles), kInferWarps * 32, smem, s>>>(params, v, warm, depth,
                                                                         W, H, nodata, threshold);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

}  // namespace cageo

using namespace cageo;

namespace {
inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }
}  // namespace

extern "C" int cageo_ws_param_count(void) { return kWsParams; }

extern "C" cageo_status cageo_ws_features(const float* d_v, float* d_feat, int W, int H, int B,
                                          float nodata_dem, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_v && d_feat && valid_dims(W, H) && B >= 1, "pointers, size and batch");
  const int64_t n = (int64_t)W * H * B;
  ws_features_kernel<<<nblk(n, 256), 256, 0, stream>>>(d_v, d_feat, W, H, B, nodata_dem);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

extern "C" cageo_status cageo_ws_infer(const float* d_params, const float* d_v, float* d_warm,
                                       float* d_depth, int W, int H, float nodata_dem,
                                       float threshold, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_params && d_v && (d_warm || d_depth) && valid_dims(W, H),
                  "pointers and size");
  return ws_infer(d_params, d_v, d_warm, d_depth, W, H, nodata_dem, threshold, stream);
}
