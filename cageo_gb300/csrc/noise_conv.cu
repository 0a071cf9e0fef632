// noise_conv.cu -- A1 Philox Gaussian noise and A3 process convolution.
//
// Convolution kernels stage a (tile + 2r halo) block of the input in shared
// memory with periodic wrap and compute every output with the reference's
// summation order (ascending taps, sum starting at 0, unfused multiply and
// add), so they equal ConvolutionAlgorithm_CPU_OpenMP bit for bit.  The
// same kernels, instantiated with the FrontEpilogue, fuse the realistic-DEM,
// burning and quantization steps of a realization into their store.
//
// What bounds them is the single-precision pipe: 2 taps products and 2 sums an
// output, each rounded on its own.  Both are issued packed, two outputs of
// neighbouring lines at a time (64-bit register pairs that the sliding windows
// never take apart), so products, sums and loads each cost half an
// instruction; results go through shared memory once more to be written in
// 16-byte pieces along the rows.
#include <algorithm>
#include <type_traits>
#include "common.cuh"
#include "f32x2.cuh"
#include "front.cuh"
#include "stage_math.cuh"

namespace cageo {

// ---- A1 ------------------------------------------------------------------
// One thread per group of 4 consecutive cells: one Philox call gives four
// uniforms -> two Box-Muller pairs -> four N(0,1) deviates.
__global__ void noise_kernel(float* __restrict__ out, int64_t n, uint32_t k0,
                             uint32_t k1, uint32_t realization,
                             const uint32_t* __restrict__ dreal, float mean,
                             float sd) {
  int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t base = g * 4;
  if (base >= n) return;
  // blockIdx.y: the field of a stack, one realization further each.
  out += blockIdx.y * n;
  realization += blockIdx.y;
  if (dreal) realization += *dreal;  // an offset from the device counter
  U4 ctr = {(uint32_t)g, realization, kNoiseTag, (uint32_t)(g >> 32)};
  U4 r = philox4x32_10(ctr, k0, k1);
  float z[4];
  {
    float rad = sqrtf(-2.0f * logf(u01_open(r.x)));
    float s, c;
    sincospif(2.0f * u01_open(r.y), &s, &c);
    z[0] = rad * c;
    z[1] = rad * s;
  }
  {
    float rad = sqrtf(-2.0f * logf(u01_open(r.z)));
    float s, c;
    sincospif(2.0f * u01_open(r.w), &s, &c);
    z[2] = rad * c;
    z[3] = rad * s;
  }
  float v[4];
#pragma unroll
  for (int j = 0; j < 4; j++) v[j] = __fadd_rn(mean, __fmul_rn(z[j], sd));
  // One float4 store when the field is 16-byte aligned (a caller's buffer
  // may start at any 4-byte boundary: then four scalar stores).
  if (base + 4 <= n && (((uintptr_t)out) & 15u) == 0) {
    *reinterpret_cast<float4*>(out + base) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
    for (int j = 0; j < 4 && base + j < n; j++) out[base + j] = v[j];
  }
}

// ---- A3 separable (Gaussian) ----------------------------------------------
// Output tile of a block (columns x rows), 256 threads.  A wider or taller
// tile stages less halo per output but leaves fewer blocks per SM, and the
// column pass (items of 8 rows x 2 columns over the tile's width plus the
// halo, 4 rows at other radii than 15 and 23) and the row pass (8 or 4 outputs
// per item, of two rows) fill the 256 threads differently for each shape and
// radius: at radius 15, 64 x 32 gives the column pass 188 items, 96 x 32 gives
// it 252.  The cageo_convolve stage
// uses the first shape; the fused front takes the pipeline's choice.
struct SepTile {
  int tw, th;
};
constexpr SepTile kSepTiles[kConvTiles] = {{64, 32}, {128, 32}, {64, 64}, {96, 32}};
constexpr int kSepThreads = 256;

// Periodic index: one period either way by compare-and-add (every index a
// valid output reads is within one period, since r < W and r < H); the
// modulo only serves padding rows/columns of very small grids.
__device__ __forceinline__ int wrap_idx(int v, int n) {
  if (v < 0) v += n;
  else if (v >= n) v -= n;
  if ((unsigned)v >= (unsigned)n) {
    v %= n;
    if (v < 0) v += n;
  }
  return v;
}

// Epilogues: what happens to the convolved values of a tile.  cell() takes one,
// quad() four along a row at once (`aligned` says that it may: the grids then
// start on 16-byte boundaries and W is a multiple of 4).  They return the least
// of the values written.
struct StoreEpilogue {
  float* out;
  bool aligned;
  __device__ __forceinline__ float cell(int64_t i, int, int, float v) const {
    out[i] = v;
    return v;
  }
  __device__ __forceinline__ float quad(int64_t i, int, int, float4 v) const {
    *reinterpret_cast<float4*>(out + i) = v;
    return 0.0f;
  }
};

// The larger value, or NaN where one of them is.
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

struct FrontEpilogue {
  FrontParams p;
  bool aligned;
  // The output grid: blockIdx.z is the grid of a stack.  (The parameters stay
  // as they are: a changed copy would live in local memory, 0.72 instead of
  // 0.58 ms at 8192^2.)
  __device__ __forceinline__ float* out() const { return p.q + blockIdx.z * ((int64_t)p.W * p.H); }
  __device__ __forceinline__ float cell(int64_t i, int x, int y, float v) const {
    const float q = front_value(p, v, p.dem[i], p.code[i]);
    out()[i] = q;
    if (front_outlet(p, x, y, q)) front_seed(p, x, y);
    return q;
  }
  __device__ __forceinline__ float quad(int64_t i, int x, int y, float4 v) const {
    const float4 d = *reinterpret_cast<const float4*>(p.dem + i);
    const unsigned int c = *reinterpret_cast<const unsigned int*>(p.code + i);
    // The common case in a few instructions a cell (70 -> 30 with the rest of the
    // epilogue, 0.60 -> 0.51 ms at 8192^2): data cells whose sums lie in
    // (0, 4000), burned or not.
    float a[4] = {__fadd_rn(d.x, v.x), __fadd_rn(d.y, v.y), __fadd_rn(d.z, v.z), __fadd_rn(d.w, v.w)};
    auto most = [&]() { return max_nan(max_nan(a[0], a[1]), max_nan(a[2], a[3])); };
    const float nd = p.nodata_dem;
    bool quick = p.quick && d.x != nd && d.y != nd && d.z != nd && d.w != nd &&
                 fminf(fminf(a[0], a[1]), fminf(a[2], a[3])) > 0.0f && most() < 4000.0f;
    if (quick) {
      bool outlet = x == 0 || y == 0 || x + 4 == p.W || y == p.H - 1;
      if (c) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const unsigned int cj = c >> 8 * j;
          if (cj & kCodeBurnStream) a[j] = 0.0f;
          if (cj & 0x1f) a[j] = __fmul_rn(a[j], p.factor[cj & 0x1f]);
        }
        quick = most() < 4000.0f && fminf(fminf(a[0], a[1]), fminf(a[2], a[3])) >= 0.0f;
      }
      if (quick) {
        float4 q = make_float4(a[0], a[1], a[2], a[3]);
        if (p.quantize)
          q = make_float4(fill_quantize_quick(a[0]), fill_quantize_quick(a[1]),
                          fill_quantize_quick(a[2]), fill_quantize_quick(a[3]));
        if (c) {  // zeros stay zeros
          if (a[0] == 0.0f) q.x = a[0], outlet = true;
          if (a[1] == 0.0f) q.y = a[1], outlet = true;
          if (a[2] == 0.0f) q.z = a[2], outlet = true;
          if (a[3] == 0.0f) q.w = a[3], outlet = true;
        }
        *reinterpret_cast<float4*>(out() + i) = q;
        if (outlet) front_seed(p, x, y);
        return fminf(fminf(q.x, q.y), fminf(q.z, q.w));
      }
    }
    float4 q;
    q.x = front_value(p, v.x, d.x, (uint8_t)c);
    q.y = front_value(p, v.y, d.y, (uint8_t)(c >> 8));
    q.z = front_value(p, v.z, d.z, (uint8_t)(c >> 16));
    q.w = front_value(p, v.w, d.w, (uint8_t)(c >> 24));
    *reinterpret_cast<float4*>(out() + i) = q;
    // (The four cells lie in one fill tile: x is a multiple of 4.)
    if (front_outlet(p, x, y, q.x) || front_outlet(p, x + 1, y, q.y) ||
        front_outlet(p, x + 2, y, q.z) || front_outlet(p, x + 3, y, q.w))
      front_seed(p, x, y);
    return fminf(fminf(q.x, q.y), fminf(q.z, q.w));
  }
};

template <class Epi>
__device__ inline void block_min_out(float local_min, const Epi&) {}

__device__ inline void block_min_out(float local_min, const FrontEpilogue& e) {
  // Block-wide min of q, then one ordered atomicMin.
  __shared__ float red[32];
  for (int o = 16; o > 0; o >>= 1)
    local_min = fminf(local_min, __shfl_xor_sync(0xffffffffu, local_min, o));
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = local_min;
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    float m = lane < nw ? red[lane] : kInf;
    for (int o = 16; o > 0; o >>= 1)
      m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0 && m < kInf) atomicMin(e.p.min_ord + blockIdx.z, float_to_ordered(m));
  }
}

// The tile's convolved values (rows of s_out, stride OS, a multiple of 4) into
// the epilogue, consecutive threads along the rows.
template <int TW, int TH, class Epi>
__device__ __forceinline__ void tile_out(const float* s_out, int OS, int x0, int y0, int W, int H,
                                         const Epi& epi) {
  float local_min = kInf;
  if (epi.aligned && x0 + TW <= W) {
    constexpr int QW = TW / 4;
#pragma unroll 2
    for (int k = threadIdx.x; k < QW * TH; k += blockDim.x) {
      const int y = k / QW, x = 4 * (k - y * QW);
      if (y0 + y >= H) break;
      const float4 v = *reinterpret_cast<const float4*>(s_out + y * OS + x);
      local_min = fminf(local_min, epi.quad((int64_t)(y0 + y) * W + x0 + x, x0 + x, y0 + y, v));
    }
  } else {
    for (int k = threadIdx.x; k < TW * TH; k += blockDim.x) {
      const int y = k / TW, x = k - y * TW;
      if (y0 + y >= H) break;
      if (x0 + x < W)
        local_min = fminf(local_min, epi.cell((int64_t)(y0 + y) * W + x0 + x, x0 + x, y0 + y,
                                              s_out[y * OS + x]));
    }
  }
  block_min_out(local_min, epi);
}

// Packed pairs of floats.  acc + w * t with the product and the sum each
// rounded to nearest (as __fmul_rn and __fadd_rn, no contraction): a packed
// multiply, and the packed sum as fma(product, 1, acc) with a 1 the compiler
// cannot see -- the assembler contracts a packed multiply feeding a packed add
// into one rounding, .rn notwithstanding; the product with 1 is exact, so this
// fused operation rounds the sum alone.
__device__ __forceinline__ f32x2 muladd2_rn(f32x2 acc, f32x2 w, f32x2 t, f32x2 one) {
  f32x2 p;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(w), "l"(t));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(p), "l"(one), "l"(acc));
  return p;
}

// N outputs (8 or 4) along a line for two neighbouring lines at once: acc[j] =
// sum_t v(j + t) * tap(t), t ascending, each sum starting at 0.  The window of N
// pairs is a ring of registers: tap t + u of a group of N finds output j's
// value at (j + u) % N and replaces entry u.  LC > 0: the tap count is a
// compile-time constant; LC = 0: runtime count L, groups of 8 taps without a
// test in between, so that their loads are in flight together.  (With a test
// at every tap, and N = 8, which leaves half of a block's threads without an
// item of the rows, a block spent most of its time on load latency: radius 64,
// 3001x401 cells, 210 us against 114; radius 30, 1500x733 cells, 34 against
// 28.5, 4096^2 cells 303 against 268.  N = 8 without the tests spills.)
template <int LC, int N, class V, class Tap>
__device__ __forceinline__ void conv_line(int L, f32x2 one, V v, Tap tap, f32x2 (&acc)[N]) {
  f32x2 win[N];
#pragma unroll
  for (int j = 0; j < N; j++) {
    win[j] = v(j);
    acc[j] = 0;
  }
  const int n = LC > 0 ? LC : L;
  auto step = [&](int t, int u) {
    const f32x2 w = tap(t);
#pragma unroll
    for (int j = 0; j < N; j++) acc[j] = muladd2_rn(acc[j], win[(j + u) & (N - 1)], w, one);
  };
  int t = 0;
  if (LC == 0) {
#pragma unroll 1
    for (; t + 8 < n; t += 8) {
#pragma unroll
      for (int u = 0; u < 8; u++) {
        step(t + u, u);
        win[u & (N - 1)] = v(t + u + N);
      }
    }
  }
#pragma unroll(LC > 0 ? (LC + 7) / 8 : 1)
  for (; t < n; t += 8) {
#pragma unroll
    for (int u = 0; u < 8; u++) {
      if (t + u < n) {
        step(t + u, u);
        if (t + u + 1 < n) win[u & (N - 1)] = v(t + u + N);
      }
    }
  }
}

// Staged columns left and right of the tile: the radius, rounded up so that
// rows start on a 16-byte boundary.
__host__ __device__ inline int sep_pad(int r) { return (r + 3) & ~3; }

// Blocks per SM the registers are held to: 5 (front at 8192^2, radius 15, 64 x
// 32 tiles, before the epilogue's quads: 0.58 ms; 4: 0.61), but 4 for radius
// 23, whose longer unrolled lines would spill (16384^2: 3.14 ms; 5: 3.27).
// 128 or 192 threads, or 6 blocks, are slower for both.  The lines are unrolled
// for these two radii (a runtime loop took 0.61 and 3.5 ms).  With the quads:
// 0.51 ms, of which the convolution alone is 0.42 and its packed products and
// sums, at two a clock and SM, 0.26.
template <class Epi, int LC, int TW, int TH>
__global__ void __launch_bounds__(kSepThreads, LC == 47 ? 4 : 5)
conv_sep_kernel(const float* __restrict__ in, int W, int H,
                const float* __restrict__ taps, int r, float one, Epi epi) {
  constexpr int N = LC > 0 ? 8 : 4;  // outputs of an item (see conv_line)
  static_assert(TW % 8 == 0 && TH % 8 == 0, "whole items");
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = 2 * r + 1, rp = sep_pad(r);
  const int IW = TW + 2 * rp, IH = TH + 2 * r, TS = IW + 1;
  f32x2* s_taps = reinterpret_cast<f32x2*>(smraw);                          // (tap, tap)
  float* s_in = reinterpret_cast<float*>(s_taps + ((L + 1) & ~1));  // IH x IW, then the outputs
  const int in_floats = IH * IW > TH * (TW + 4) ? IH * IW : TH * (TW + 4);
  f32x2* s_tmp = reinterpret_cast<f32x2*>(s_in + in_floats);        // TH/2 x TS: rows 2j, 2j + 1
  const int x0 = blockIdx.x * TW, y0 = blockIdx.y * TH;
  in += blockIdx.z * (int64_t)W * H;  // a field of a stack
  const f32x2 one2 = pack2(one, one);
  for (int t = threadIdx.x; t < L; t += kSepThreads) {
    const float v = taps[t];
    s_taps[t] = pack2(v, v);
  }
  if (x0 >= rp && x0 + TW + rp <= W && (W & 3) == 0 && ((uintptr_t)in & 15u) == 0) {
    // No column wraps: 16-byte copies.
    const int CW = IW / 4;
    int iy = threadIdx.x / CW, ic = threadIdx.x - iy * CW;
    const int dy = kSepThreads / CW, dc = kSepThreads - dy * CW;
#pragma unroll 2
    for (int k = threadIdx.x; k < IH * CW; k += kSepThreads) {
      const int gy = wrap_idx(y0 - r + iy, H);
      cp_async16(s_in + 4 * k, in + (int64_t)gy * W + x0 - rp + 4 * ic);
      iy += dy;
      ic += dc;
      if (ic >= CW) {
        ic -= CW;
        iy++;
      }
    }
  } else {
    int iy = threadIdx.x / IW, ix = threadIdx.x - iy * IW;
    const int dy = kSepThreads / IW, dx = kSepThreads - dy * IW;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < IW * IH; idx += kSepThreads) {
      const int gy = wrap_idx(y0 - r + iy, H), gx = wrap_idx(x0 - rp + ix, W);
      cp_async4(&s_in[idx], &in[(int64_t)gy * W + gx]);  // all of them in flight at once
      iy += dy;
      ix += dx;
      if (ix >= IW) {
        ix -= IW;
        iy++;
      }
    }
  }
  cp_async_wait();
  __syncthreads();
  // Column pass: tmp[y][ix] = sum_t in[y+t][ix] * taps[t]; an item is N rows
  // of two adjacent columns.  The results are kept as pairs of rows, which is
  // what the row pass multiplies; its row stride is odd, so 16 row pairs are
  // read without bank conflicts.
  const int p0 = (rp - r) >> 1, np = ((rp + TW + r + 1) >> 1) - p0;
  for (int item = threadIdx.x; item < np * (TH / N); item += kSepThreads) {
    const int g = item / np, ix = 2 * (p0 + item - g * np);
    const float* base = s_in + (N * g) * IW + ix;
    f32x2 acc[N];
    conv_line<LC, N>(L, one2,
                     [&](int k) { return *reinterpret_cast<const f32x2*>(base + k * IW); },
                     [&](int t) { return s_taps[t]; }, acc);
#pragma unroll
    for (int j = 0; j < N / 2; j++) {
      float a0, a1, b0, b1;
      unpack2(acc[2 * j], a0, a1);
      unpack2(acc[2 * j + 1], b0, b1);
      f32x2* o = s_tmp + (N / 2 * g + j) * TS + ix;
      o[0] = pack2(a0, b0);
      o[1] = pack2(a1, b1);
    }
  }
  __syncthreads();
  // Row pass: an item is N consecutive outputs of two rows.
  constexpr int OS = TW + 4;
  float* s_out = s_in;
  for (int item = threadIdx.x; item < (TH / 2) * (TW / N); item += kSepThreads) {
    const int g = item / (TH / 2), j = item - g * (TH / 2);
    const f32x2* base = s_tmp + j * TS + N * g + (rp - r);
    f32x2 acc[N];
    conv_line<LC, N>(L, one2, [&](int k) { return base[k]; }, [&](int t) { return s_taps[t]; }, acc);
    float* o = s_out + 2 * j * OS + N * g;
#pragma unroll
    for (int k = 0; k < N; k++) unpack2(acc[k], o[k], o[OS + k]);
  }
  __syncthreads();
  tile_out<TW, TH>(s_out, OS, x0, y0, W, H, epi);
}

// ---- A3 full 2D (exponential) -----------------------------------------------
// A block computes a 64 x TH tile; a thread 8 consecutive outputs of rows j and
// j + TH/2 as packed pairs from a sliding window.  PAIRED: the input is staged
// as those pairs and the taps twice, so a tap costs one load of input and one
// broadcast load of the tap per 16 outputs; larger filters, whose pairs would
// not fit shared memory, load the two rows and pack the tap.  Lane = row, and
// the row stride is odd: no bank conflicts.
// Each output's sum runs over the filter rows, and inside a row over its taps,
// in ascending order, as the reference's 2D loop does.  TH = 64 where the grid
// then still has 8 tiles per SM to balance; 32 otherwise.
constexpr int kTwoDTW = 64;
constexpr int kTwoDBlocks = 8 * 152;
constexpr int kTwoDPairedRadius = 31;

template <class Epi, int TH, bool PAIRED>
__global__ void __launch_bounds__(4 * TH)
conv_2d_kernel(const float* __restrict__ in, int W, int H,
               const float* __restrict__ filt, int r, float one, Epi epi) {
  constexpr int NT = 4 * TH, NP = TH / 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int L = 2 * r + 1;
  const int IW = kTwoDTW + 2 * r, IH = TH + 2 * r, S = IW | 1;
  float* s_f = reinterpret_cast<float*>(smraw);
  f32x2* s_f2 = reinterpret_cast<f32x2*>(smraw);
  unsigned char* rows = smraw + sizeof(float) * (((PAIRED ? 2 : 1) * L * L + 3) & ~3);
  f32x2* s_in2 = reinterpret_cast<f32x2*>(rows);  // PAIRED: rows y, y + NP
  float* s_in = reinterpret_cast<float*>(rows);
  const f32x2 one2 = pack2(one, one);
  const int x0 = blockIdx.x * kTwoDTW, y0 = blockIdx.y * TH;
  in += blockIdx.z * (int64_t)W * H;  // a field of a stack
  for (int t = threadIdx.x; t < L * L; t += NT) {
    const float v = filt[t];
    if (PAIRED) s_f2[t] = pack2(v, v);
    else s_f[t] = v;
  }
  {
    int iy = threadIdx.x / IW, ix = threadIdx.x - iy * IW;
    const int dy = NT / IW, dx = NT - dy * IW;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < IW * IH; idx += NT) {
      const int gy = wrap_idx(y0 - r + iy, H), gx = wrap_idx(x0 - r + ix, W);
      const float* src = &in[(int64_t)gy * W + gx];
      if (PAIRED) {  // all of them in flight at once
        float* d = reinterpret_cast<float*>(s_in2 + iy * S + ix);
        if (iy < NP + 2 * r) cp_async4(d, src);
        if (iy >= NP) cp_async4(d - 2 * NP * S + 1, src);
      } else {
        cp_async4(&s_in[iy * S + ix], src);
      }
      iy += dy;
      ix += dx;
      if (ix >= IW) {
        ix -= IW;
        iy++;
      }
    }
    cp_async_wait();
  }
  __syncthreads();
  const int j = threadIdx.x % NP, g = threadIdx.x / NP;
  f32x2 acc[8];
#pragma unroll
  for (int k = 0; k < 8; k++) acc[k] = 0;
  for (int fy = 0; fy < L; fy++) {
    const int f = fy * L, o = (j + fy) * S + 8 * g;
    auto tap = [&](int t) { return PAIRED ? s_f2[f + t] : pack2(s_f[f + t], s_f[f + t]); };
    auto value = [&](int k) { return PAIRED ? s_in2[o + k] : pack2(s_in[o + k], s_in[o + NP * S + k]); };
    f32x2 win[8];
#pragma unroll
    for (int k = 0; k < 8; k++) win[k] = value(k);
    int t = 0;
#pragma unroll 1
    for (; t + 8 < L; t += 8) {
#pragma unroll
      for (int u = 0; u < 8; u++) {
        const f32x2 w = tap(t + u);
#pragma unroll
        for (int k = 0; k < 8; k++) acc[k] = muladd2_rn(acc[k], win[(k + u) & 7], w, one2);
        win[u] = value(t + u + 8);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; u++) {
      if (t + u >= L) break;
      const f32x2 w = tap(t + u);
#pragma unroll
      for (int k = 0; k < 8; k++) acc[k] = muladd2_rn(acc[k], win[(k + u) & 7], w, one2);
      if (t + u + 1 < L) win[u] = value(t + u + 8);
    }
  }
  __syncthreads();
  constexpr int OS = kTwoDTW + 4;
  float* s_out = s_in;
#pragma unroll
  for (int k = 0; k < 8; k++)
    unpack2(acc[k], s_out[j * OS + 8 * g + k], s_out[(j + NP) * OS + 8 * g + k]);
  __syncthreads();
  tile_out<kTwoDTW, TH>(s_out, OS, x0, y0, W, H, epi);
}

size_t conv_2d_smem_bytes(int r, int th) {
  const int L = 2 * r + 1, S = (kTwoDTW + 2 * r) | 1;
  const bool paired = r <= kTwoDPairedRadius;
  return sizeof(float) * ((((paired ? 2 : 1) * L * L + 3) & ~3) +
                          std::max((size_t)(paired ? th + 4 * r : th + 2 * r) * S,
                                   (size_t)th * (kTwoDTW + 4)));
}

size_t conv_smem_bytes(int model, int r, int tile) {
  if (model != CAGEO_FILTER_GAUSSIAN) return conv_2d_smem_bytes(r, 32);
  const int L = 2 * r + 1;
  const SepTile t = kSepTiles[tile];
  const int IW = t.tw + 2 * sep_pad(r), IH = t.th + 2 * r;
  return sizeof(float) * (2 * ((L + 1) & ~1) +
                          std::max((size_t)IW * IH, (size_t)t.th * (t.tw + 4)) +
                          (size_t)t.th * (IW + 1));
}

// Whether a tile shape of the fused front applies: Gaussian filters (the
// separable kernel) whose staged block fits the device's shared memory.
bool conv_tile_applies(int model, int r, int tile) {
  if (model != CAGEO_FILTER_GAUSSIAN || tile < 0 || tile >= kConvTiles) return tile == 0;
  int optin = 0, dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return tile == 0;
  // The kernels' own static shared memory (the block minimum) is small.
  return conv_smem_bytes(model, r, tile) + 1024 <= (size_t)optin;
}

// The separable kernel for a tile shape and radius: fully unrolled for the
// 60 m and 90 m ranges at 10 m cells (radius 15 and 23).
template <class Epi>
using SepKernel = void (*)(const float*, int, int, const float*, int, float, Epi);

template <class Epi, int TW, int TH>
SepKernel<Epi> sep_kernel_for(int r) {
  return r == 15 ? conv_sep_kernel<Epi, 31, TW, TH>
                 : r == 23 ? conv_sep_kernel<Epi, 47, TW, TH> : conv_sep_kernel<Epi, 0, TW, TH>;
}

template <class Epi>
SepKernel<Epi> sep_kernel(int r, int tile) {
  if constexpr (std::is_same<Epi, FrontEpilogue>::value) {
    switch (tile) {
      case 1: return sep_kernel_for<Epi, kSepTiles[1].tw, kSepTiles[1].th>(r);
      case 2: return sep_kernel_for<Epi, kSepTiles[2].tw, kSepTiles[2].th>(r);
      case 3: return sep_kernel_for<Epi, kSepTiles[3].tw, kSepTiles[3].th>(r);
      default: break;
    }
  }
  return sep_kernel_for<Epi, kSepTiles[0].tw, kSepTiles[0].th>(r);
}

template <class Epi>
cageo_status launch_conv(const float* in, int W, int H, int model,
                         const float* filt, int r, const Epi& epi,
                         cudaStream_t s, int tile = 0, int slabs = 1) {
  if (!std::is_same<Epi, FrontEpilogue>::value || tile < 0 || tile >= kConvTiles) tile = 0;
  // The kernels' dynamic shared-memory limit is raised to the most the
  // device allows (its opt-in maximum less the kernel's static shared
  // memory), the same value on every call: pipelines on other host threads
  // launch the same kernels with other radii, and a per-call limit set by
  // one thread could fall below another thread's launch between its set
  // and launch.  (Occupancy follows each launch's own size, not the limit.)
  int optin = 0, dev = 0;
  CAGEO_CUDA(cudaGetDevice(&dev));
  CAGEO_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  auto raise_limit = [&](const void* fn, int* limit) -> cageo_status {
    cudaFuncAttributes fa;
    CAGEO_CUDA(cudaFuncGetAttributes(&fa, fn));
    *limit = optin - (int)fa.sharedSizeBytes;
    CAGEO_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, *limit));
    return CAGEO_OK;
  };
  if (model == CAGEO_FILTER_GAUSSIAN) {
    const size_t smem = conv_smem_bytes(model, r, tile);
    const SepKernel<Epi> fn = sep_kernel<Epi>(r, tile);
    int limit = 0;
    cageo_status st = raise_limit((const void*)fn, &limit);
    if (st) return st;
    if (smem > (size_t)limit) {
      set_error("filter radius %d needs %zu bytes of shared memory (%d available)", r, smem, limit);
      return CAGEO_ERR_ARGUMENT;
    }
    const SepTile t = kSepTiles[tile];
    dim3 grid((W + t.tw - 1) / t.tw, (H + t.th - 1) / t.th, slabs);
    fn<<<grid, kSepThreads, smem, s>>>(in, W, H, filt, r, 1.0f, epi);
  } else {
    using Kernel = SepKernel<Epi>;
    const bool paired = r <= kTwoDPairedRadius;
    const int gx = (W + kTwoDTW - 1) / kTwoDTW;
    int th = (int64_t)slabs * gx * ((H + 63) / 64) >= kTwoDBlocks ? 64 : 32, limit = 0;
    for (;; th = 32) {
      const Kernel fn = th == 64 ? (paired ? (Kernel)conv_2d_kernel<Epi, 64, true>
                                        : (Kernel)conv_2d_kernel<Epi, 64, false>)
                                 : (paired ? (Kernel)conv_2d_kernel<Epi, 32, true>
                                        : (Kernel)conv_2d_kernel<Epi, 32, false>);
      cageo_status st = raise_limit((const void*)fn, &limit);
      if (st) return st;
      const size_t bytes = conv_2d_smem_bytes(r, th);
      if (bytes > (size_t)limit && th == 64) continue;
      if (bytes > (size_t)limit) {
        set_error("filter radius %d needs %zu bytes of shared memory (%d available)", r, bytes, limit);
        return CAGEO_ERR_ARGUMENT;
      }
      fn<<<dim3(gx, (H + th - 1) / th, slabs), 4 * th, bytes, s>>>(in, W, H, filt, r, 1.0f, epi);
      break;
    }
  }
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

cageo_status launch_noise(float* d, int64_t n, uint64_t seed, uint32_t realization,
                          const uint32_t* dreal, float mean, float sd, cudaStream_t s, int slabs) {
  int64_t groups = (n + 3) / 4;
  int threads = 256;
  int64_t blocks = (groups + threads - 1) / threads;
  noise_kernel<<<dim3((unsigned)blocks, slabs), threads, 0, s>>>(d, n, (uint32_t)seed,
                                                    (uint32_t)(seed >> 32), realization,
                                                    dreal, mean, sd);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

cageo_status launch_front(const float* noise, int W, int H, int model,
                          const float* filt, int r, const FrontParams& fp,
                          cudaStream_t s, int tile, int slabs) {
  const uintptr_t ptrs = (uintptr_t)fp.dem | (uintptr_t)fp.q;
  FrontEpilogue e{fp, (W & 3) == 0 && (ptrs & 15u) == 0 && ((uintptr_t)fp.code & 3u) == 0};
  return launch_conv(noise, W, H, model, filt, r, e, s, tile, slabs);
}

}  // namespace cageo

using namespace cageo;

extern "C" cageo_status cageo_noise_philox(float* d_field, int W, int H,
                                           uint64_t seed, uint32_t realization,
                                           float mean, float stddev,
                                           cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_field && valid_dims(W, H), "field pointer and size");
  return launch_noise(d_field, (int64_t)W * H, seed, realization, nullptr, mean, stddev, stream,
                      1);
}

// Raw Philox4x32-10 blocks: block i is philox4x32_10((c0 + i, c1, c2, c3),
// (k0, k1)), the generator noise_kernel draws from.
__global__ void philox_bits_kernel(uint32_t* __restrict__ out, int64_t n, U4 c, uint32_t k0,
                                   uint32_t k1) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  U4 ci = c;
  ci.x += (uint32_t)i;
  const U4 r = philox4x32_10(ci, k0, k1);
  out[4 * i] = r.x;
  out[4 * i + 1] = r.y;
  out[4 * i + 2] = r.z;
  out[4 * i + 3] = r.w;
}

extern "C" cageo_status cageo_philox4x32_10(uint32_t* d_out, int64_t n, const uint32_t* h_ctr,
                                            const uint32_t* h_key, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_out && h_ctr && h_key && n > 0 && n < ((int64_t)1 << 31),
                  "pointers and block count");
  const U4 c = {h_ctr[0], h_ctr[1], h_ctr[2], h_ctr[3]};
  philox_bits_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(d_out, n, c, h_key[0],
                                                                      h_key[1]);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

extern "C" cageo_status cageo_convolve(const float* d_in, float* d_out, int W,
                                       int H, int model, const float* d_filter,
                                       int radius, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_in && d_out && d_filter && valid_dims(W, H), "pointers and size");
  CAGEO_CHECK_ARG(d_in != d_out, "convolution cannot run in place");
  CAGEO_CHECK_ARG(model == CAGEO_FILTER_GAUSSIAN || model == CAGEO_FILTER_EXPONENTIAL,
                  "filter model");
  CAGEO_CHECK_ARG(radius >= 0 && radius < W && radius < H,
                  "filter radius must be below the grid width and height");
  StoreEpilogue e{d_out, (W & 3) == 0 && ((uintptr_t)d_out & 15u) == 0};
  return launch_conv(d_in, W, H, model, d_filter, radius, e, stream);
}
