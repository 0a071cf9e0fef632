// learned_train.cu -- training of the learned warm start's network (no
// counterpart in the reference): forward pass, gradients of every parameter,
// mean-squared-error loss, Adam.  fp32 on the CUDA cores, weights rounded to
// bf16 where they are used, activations planar [batch][channel][H][W].
//
// The three 3x3 convolutions between 32 channels (forward, input gradient,
// weight gradient of layer 2) are nearly all of the work: 2.4 G multiply-adds
// each for 16 grids of 128x128, 60 us at the fp32 rate.  All kernels keep a
// tile of inputs in shared memory and a block of results in registers, so
// that a loaded value serves 16 to 72 multiply-adds, two per instruction.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <initializer_list>
#include <type_traits>
#include "f32x2.cuh"
#include "learned.cuh"

namespace cageo {

constexpr int kTrainThreads = 128;

template <int N>
__device__ __forceinline__ void cp_async_wait_all_but() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// The grids of a batch cut into tiles of 32 columns and `rows` rows.
struct TrainTiles {
  int W, H, tiles_x, tiles_y;
  int64_t count;
  __host__ __device__ TrainTiles(int W, int H, int B, int rows)
      : W(W), H(H), tiles_x((W + 31) / 32), tiles_y((H + rows - 1) / rows),
        count((int64_t)tiles_x * tiles_y * B) {}
  __device__ void at(int64_t tile, int rows, int& b, int& x0, int& y0) const {
    const int64_t r = tile / tiles_x;
    x0 = (int)(tile - r * tiles_x) * 32;
    b = (int)(r / tiles_y);
    y0 = (int)(r - (int64_t)b * tiles_y) * rows;
  }
};

// ---- convolution to 32 channels ------------------------------------------------
// out[b][co](y,x) = bias[co] + sum_ci sum_t w[co][ci][t] * in[b][ci](y+dy, x+dx),
// zero outside, each sum in that order from the bias on; then the optional
// ReLU, and 0 where mask is not positive (the ReLU's gradient, mask: its
// output).  FLIP: w holds the weights of the convolution whose input gradient
// this is, [ci][co][8 - t].
//
// A thread has 4 cells of a row and 8 output channels; the 4 warps of a block
// take the 4 channel groups of a 32x4 tile, so the weights (pairs of channels)
// are read by broadcast.  A staged row is kept as its four residues of the
// column mod 4, 10 apart, 40 a row: the 32 lanes' cells (8 of a row, 4 rows)
// then lie in 32 banks.  The channels arrive in two halves, the next tile's
// while the other half is worked on.  Three blocks an SM hold their weights
// over all their tiles.
// Bound by the fp32 rate: 0.13 ms between 32 channels for 16 x 128x128 (0.20
// with one cell and all channels a thread, a scalar weight load per product).
constexpr int kConvRows = 4;
constexpr int kResidue = 10, kInRow = 4 * kResidue, kInPlane = (kConvRows + 2) * kInRow;
constexpr int kWeightRow = 36;  // 32 channels of a (ci, t), padded against store conflicts

size_t conv32_smem(int cin) { return (size_t)cin * (9 * kWeightRow + kInPlane) * sizeof(float); }

template <bool FLIP>
__global__ void __launch_bounds__(kTrainThreads, 3)
train_conv32_kernel(const float* __restrict__ in, int cin, const float* __restrict__ w,
                    const float* __restrict__ bias, const float* __restrict__ mask,
                    float* __restrict__ out, int W, int H, int B, int relu, int vec) {
  extern __shared__ __align__(16) float smem[];
  float* sw = smem;                          // [ci][t][co]
  float* sa = smem + cin * 9 * kWeightRow;   // [ci][row][residue][column / 4]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t n = (int64_t)W * H;
  const TrainTiles tiles(W, H, B, kConvRows);
  const int half = (cin + 1) / 2;

  auto stage = [&](int64_t tile, int c0, int c1) {
    if (tile < tiles.count) {
      int b, x0, y0;
      tiles.at(tile, kConvRows, b, x0, y0);
      const float* src = in + (int64_t)b * cin * n;
      auto copy = [&](int rr, int slot) {  // slot: column x0 - 1 + slot
        const int ci = rr / (kConvRows + 2), row = rr - ci * (kConvRows + 2);
        const int x = x0 - 1 + slot, y = y0 - 1 + row;
        float* d = sa + ci * kInPlane + row * kInRow + (slot & 3) * kResidue + (slot >> 2);
        if (x >= 0 && x < W && y >= 0 && y < H) cp_async4(d, src + ci * n + (int64_t)y * W + x);
        else *d = 0.0f;
      };
      for (int rr = c0 * (kConvRows + 2) + warp; rr < c1 * (kConvRows + 2); rr += 4)
        copy(rr, lane + 1);
      for (int k = c0 * 2 * (kConvRows + 2) + tid; k < c1 * 2 * (kConvRows + 2); k += kTrainThreads)
        copy(k >> 1, (k & 1) * 33);
    }
    cp_async_commit();
  };
  stage(blockIdx.x, 0, half);
  stage(blockIdx.x, half, cin);
  bool odd = false;  // a weight that is infinite or NaN: zero padding would not be neutral
  for (int k = tid; k < 32 * cin * 9; k += kTrainThreads) {
    int co, r;  // r = ci * 9 + t
    if (FLIP) {
      const int ci = k / 288, m = k - ci * 288;
      co = m / 9;
      r = ci * 9 + 8 - (m - co * 9);
    } else {
      co = k / (cin * 9);
      r = k - co * cin * 9;
    }
    const float v = bf16_round(w[k]);
    odd |= !isfinite(v);
    sw[r * kWeightRow + co] = v;
  }
  const bool guard = __syncthreads_or(odd);

  const int ly = lane >> 3, g = lane & 7, co0 = warp * 8;
  f32x2 first[4];
#pragma unroll
  for (int k = 0; k < 4; k++)
    first[k] = bias ? pack2(bf16_round(bias[co0 + 2 * k]), bf16_round(bias[co0 + 2 * k + 1])) : 0;
  for (int64_t tile = blockIdx.x; tile < tiles.count; tile += gridDim.x) {
    int b, x0, y0;
    tiles.at(tile, kConvRows, b, x0, y0);
    const int x = x0 + 4 * g, y = y0 + ly;
    f32x2 acc[4][4];  // [cell][pair of channels]
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int k = 0; k < 4; k++) acc[j][k] = first[k];
    auto sums = [&](auto guarded, int c0, int c1) {
#pragma unroll 1
      for (int ci = c0; ci < c1; ci++) {
        const float* base = sa + ci * kInPlane + ly * kInRow + g;
        const float* wt = sw + ci * 9 * kWeightRow + co0;
#pragma unroll
        for (int dy = 0; dy < 3; dy++) {
          f32x2 a[6];
#pragma unroll
          for (int j = 0; j < 6; j++) {
            const float v = base[dy * kInRow + (j & 3) * kResidue + (j >> 2)];
            a[j] = pack2(v, v);
          }
#pragma unroll
          for (int dx = 0; dx < 3; dx++) {
            const float* p = wt + (dy * 3 + dx) * kWeightRow;
            const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(p);
            const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(p + 4);
#pragma unroll
            for (int j = 0; j < 4; j++) {
              if constexpr (decltype(guarded)::value) {
                const int xx = x + j + dx - 1, yy = y + dy - 1;
                if (xx < 0 || yy < 0 || xx >= W || yy >= H) continue;
              }
              acc[j][0] = fma2(w0.x, a[j + dx], acc[j][0]);
              acc[j][1] = fma2(w0.y, a[j + dx], acc[j][1]);
              acc[j][2] = fma2(w1.x, a[j + dx], acc[j][2]);
              acc[j][3] = fma2(w1.y, a[j + dx], acc[j][3]);
            }
          }
        }
      }
    };
    auto compute = [&](int c0, int c1) {
      if (guard) sums(std::true_type(), c0, c1);
      else sums(std::false_type(), c0, c1);
    };
    const int64_t next = tile + gridDim.x;
    cp_async_wait_all_but<1>();
    __syncthreads();
    compute(0, half);
    __syncthreads();
    stage(next, 0, half);
    cp_async_wait_all_but<1>();
    __syncthreads();
    compute(half, cin);
    __syncthreads();
    stage(next, half, cin);
    if (x >= W || y >= H) continue;  // (no barrier is skipped)
    const int64_t o = ((int64_t)b * 32 + co0) * n + (int64_t)y * W + x;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float lo, hi;
        unpack2(acc[j][k >> 1], lo, hi);
        v[j] = k & 1 ? hi : lo;
        if (relu) v[j] = fmaxf(v[j], 0.0f);
      }
      float* d = out + o + k * n;
      const float* m = mask ? mask + o + k * n : nullptr;
      if (vec) {
        if (m) {
          const float4 f = *reinterpret_cast<const float4*>(m);
          if (!(f.x > 0.0f)) v[0] = 0.0f;
          if (!(f.y > 0.0f)) v[1] = 0.0f;
          if (!(f.z > 0.0f)) v[2] = 0.0f;
          if (!(f.w > 0.0f)) v[3] = 0.0f;
        }
        *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (x + j < W) d[j] = m && !(m[j] > 0.0f) ? 0.0f : v[j];
      }
    }
  }
}

// ---- convolution of 32 channels to one -------------------------------------------
// The network's output layer: the same sums, one cell a thread.  Bound by the
// read of the 32 channels and the 9 shared loads a channel.
constexpr int kOneRow = 36, kOnePlane = (kConvRows + 2) * kOneRow;

__global__ void __launch_bounds__(kTrainThreads)
train_conv1_kernel(const float* __restrict__ in, const float* __restrict__ w,
                   const float* __restrict__ bias, float* __restrict__ out, int W, int H, int B) {
  __shared__ __align__(16) float sw[32 * 12];
  __shared__ float sa[32 * kOnePlane];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t n = (int64_t)W * H;
  const TrainTiles tiles(W, H, B, kConvRows);
  auto stage = [&](int64_t tile, int c0, int c1) {
    if (tile < tiles.count) {
      int b, x0, y0;
      tiles.at(tile, kConvRows, b, x0, y0);
      const float* src = in + (int64_t)b * 32 * n;
      auto copy = [&](int rr, int slot) {
        const int ci = rr / (kConvRows + 2), row = rr - ci * (kConvRows + 2);
        const int x = x0 - 1 + slot, y = y0 - 1 + row;
        float* d = sa + rr * kOneRow + slot;
        if (x >= 0 && x < W && y >= 0 && y < H) cp_async4(d, src + ci * n + (int64_t)y * W + x);
        else *d = 0.0f;
      };
      for (int rr = c0 * (kConvRows + 2) + warp; rr < c1 * (kConvRows + 2); rr += 4)
        copy(rr, lane + 1);
      for (int k = c0 * 2 * (kConvRows + 2) + tid; k < c1 * 2 * (kConvRows + 2); k += kTrainThreads)
        copy(k >> 1, (k & 1) * 33);
    }
    cp_async_commit();
  };
  stage(blockIdx.x, 0, 16);
  stage(blockIdx.x, 16, 32);
  bool odd = false;
  for (int k = tid; k < 288; k += kTrainThreads) {
    const float v = bf16_round(w[k]);
    odd |= !isfinite(v);
    sw[k / 9 * 12 + k % 9] = v;
  }
  const bool guard = __syncthreads_or(odd);
  const float first = bias ? bf16_round(*bias) : 0.0f;
  for (int64_t tile = blockIdx.x; tile < tiles.count; tile += gridDim.x) {
    int b, x0, y0;
    tiles.at(tile, kConvRows, b, x0, y0);
    const int x = x0 + lane, y = y0 + warp;
    float acc = first;
    auto sums = [&](auto guarded, int c0, int c1) {
#pragma unroll 4
      for (int ci = c0; ci < c1; ci++) {
        const float4 wa = *reinterpret_cast<const float4*>(sw + ci * 12);
        const float4 wb = *reinterpret_cast<const float4*>(sw + ci * 12 + 4);
        const float wt[9] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w, sw[ci * 12 + 8]};
#pragma unroll
        for (int t = 0; t < 9; t++) {
          if constexpr (decltype(guarded)::value) {
            const int xx = x + t % 3 - 1, yy = y + t / 3 - 1;
            if (xx < 0 || yy < 0 || xx >= W || yy >= H) continue;
          }
          acc = fmaf(wt[t], sa[ci * kOnePlane + (warp + t / 3) * kOneRow + lane + t % 3], acc);
        }
      }
    };
    auto compute = [&](int c0, int c1) {
      if (guard) sums(std::true_type(), c0, c1);
      else sums(std::false_type(), c0, c1);
    };
    const int64_t next = tile + gridDim.x;
    cp_async_wait_all_but<1>();
    __syncthreads();
    compute(0, 16);
    __syncthreads();
    stage(next, 0, 16);
    cp_async_wait_all_but<1>();
    __syncthreads();
    compute(16, 32);
    __syncthreads();
    stage(next, 16, 32);
    if (x < W && y < H) out[(int64_t)b * n + (int64_t)y * W + x] = acc;
  }
}

// ---- grids a few cells wide ------------------------------------------------------
// The same sums with one cell and COUT channels a thread, in the same order: the
// tiles above are 32 columns wide whatever the grid is.
template <int COUT, bool FLIP>
__global__ void __launch_bounds__(kTrainThreads)
train_conv_narrow_kernel(const float* __restrict__ in, int cin, const float* __restrict__ w,
                         const float* __restrict__ bias, const float* __restrict__ mask,
                         float* __restrict__ out, int W, int H, int B, int relu) {
  extern __shared__ __align__(16) float smem[];  // [ci][t][co]
  for (int k = threadIdx.x; k < COUT * cin * 9; k += kTrainThreads) {
    const int t = k % 9, p = k / 9;  // FLIP: [ci][co][8 - t], otherwise [co][ci][t]
    const int ci = FLIP ? p / COUT : p % cin, co = FLIP ? p % COUT : p / cin;
    smem[(ci * 9 + (FLIP ? 8 - t : t)) * COUT + co] = bf16_round(w[k]);
  }
  __syncthreads();
  const int64_t n = (int64_t)W * H, i = (int64_t)blockIdx.x * kTrainThreads + threadIdx.x;
  if (i >= n * B) return;
  const int b = (int)(i / n);
  const int64_t c = i - (int64_t)b * n;
  const int x = (int)(c % W), y = (int)(c / W);
  float acc[COUT];
#pragma unroll
  for (int co = 0; co < COUT; co++) acc[co] = bias ? bf16_round(bias[co]) : 0.0f;
  for (int ci = 0; ci < cin; ci++) {
    const float* plane = in + ((int64_t)b * cin + ci) * n;
#pragma unroll
    for (int t = 0; t < 9; t++) {
      const int xx = x + t % 3 - 1, yy = y + t / 3 - 1;
      if (xx < 0 || yy < 0 || xx >= W || yy >= H) continue;
      const float a = plane[(int64_t)yy * W + xx];
#pragma unroll
      for (int co = 0; co < COUT; co++) acc[co] = fmaf(smem[(ci * 9 + t) * COUT + co], a, acc[co]);
    }
  }
  const int64_t o = (int64_t)b * COUT * n + c;
#pragma unroll
  for (int co = 0; co < COUT; co++) {
    float v = relu ? fmaxf(acc[co], 0.0f) : acc[co];
    if (mask && !(mask[o + co * n] > 0.0f)) v = 0.0f;
    out[o + co * n] = v;
  }
}

// Weight gradients of such grids: a block per output channel and input channel.
__global__ void __launch_bounds__(256)
train_wgrad_narrow_kernel(const float* __restrict__ dz, int cout, const float* __restrict__ a,
                          int cin, float* __restrict__ gw, float* __restrict__ gb, int W, int H,
                          int B) {
  const int co = blockIdx.x / cin, ci = blockIdx.x % cin;
  const int64_t n = (int64_t)W * H;
  float s[10] = {};
  for (int64_t i = threadIdx.x; i < n * B; i += 256) {
    const int b = (int)(i / n);
    const int64_t c = i - (int64_t)b * n;
    const float g = dz[((int64_t)b * cout + co) * n + c];
    if (g == 0.0f) continue;
    const float* p = a + ((int64_t)b * cin + ci) * n;
    const int x = (int)(c % W), y = (int)(c / W);
#pragma unroll
    for (int t = 0; t < 9; t++) {
      const int xx = x + t % 3 - 1, yy = y + t / 3 - 1;
      if (xx < 0 || yy < 0 || xx >= W || yy >= H) continue;
      s[t] = fmaf(g, p[(int64_t)yy * W + xx], s[t]);
    }
    s[9] += g;
  }
  __shared__ float red[8][10];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int t = 0; t < 10; t++) {
    float v = s[t];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp][t] = v;
  }
  __syncthreads();
  if (threadIdx.x < 10) {
    float v = 0.0f;
    for (int k = 0; k < 8; k++) v += red[k][threadIdx.x];
    if (threadIdx.x < 9) gw[(co * cin + ci) * 9 + threadIdx.x] += v;
    else if (ci == 0) gb[co] += v;
  }
}

// ---- weight gradients ---------------------------------------------------------
// gw[co][ci][t] += sum_b sum_cell dz[b][co](y,x) * a[b][ci](y+dy, x+dx) and
// gb[co] += sum dz[b][co].
//
// A block walks over tiles of 32 columns and ROWS rows with all channels of
// both grids in shared memory (two buffers: the next tile arrives meanwhile),
// dz with its channels innermost.  A thread keeps the 9 taps of TCO x 2 channel
// pairs in registers, two output channels to a register pair: 144 packed
// multiply-adds for 10 16-byte loads (TCO = 4).  Layers with fewer channels
// split the tile's rows over PXS lanes instead.  Each block's sums go to `part`
// and train_wsum_kernel adds them in a fixed order; a single block adds to the
// gradients itself.
// A product of zero and an infinite value or a NaN is left out by definition
// (padding, cells without gradient), which plain sums do not do: where a sum
// comes out infinite or NaN the block's tiles are summed again cell by cell.
// Bound by the fp32 rate: layer 2 takes 0.12 ms for 16 x 128x128 (1.9 with a
// block per channel pair, 20 times the reads and most of its loads re-read).
constexpr int kARow = 44;  // columns -1..32 at 3..36

template <int COUT, int TCO, int CIG, int PXS, int ROWS>
struct Wgrad {
  static constexpr int kCog = (COUT + TCO - 1) / TCO, kCin = 2 * CIG;
  // Strides that keep the lanes' loads in different banks.
  static constexpr int kAPlane = (ROWS + 2) * kARow + 4;
  static constexpr int kDCell = COUT == 1 ? 2 : COUT + 4, kDRow = 32 * kDCell + 4;
  static constexpr int kBuf = kCin * kAPlane + ROWS * kDRow;
  static constexpr int kWeights = COUT * kCin * 9, kSums = kWeights + COUT;
  static constexpr int kSmem = 2 * kBuf * (int)sizeof(float);
  static_assert(kCog * CIG * PXS == kTrainThreads && ROWS % PXS == 0, "one thread per part");
  static_assert(TCO % 2 == 0 && (COUT == 1 || COUT % TCO == 0), "pairs of output channels");
};

template <int COUT, int TCO, int CIG, int PXS, int ROWS>
__global__ void __launch_bounds__(kTrainThreads, 3)
train_wgrad_kernel(const float* __restrict__ dz, const float* __restrict__ a, float* __restrict__ gw,
                   float* __restrict__ gb, float* __restrict__ part, int W, int H, int B, int vec) {
  using G = Wgrad<COUT, TCO, CIG, PXS, ROWS>;
  extern __shared__ __align__(16) float smem[];
  __shared__ float s_bias[4 * COUT];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t n = (int64_t)W * H;
  const TrainTiles tiles(W, H, B, ROWS);
  if (COUT == 1) {  // the pair's other half
    for (int k = tid; k < 2 * G::kBuf; k += kTrainThreads) smem[k] = 0.0f;
    __syncthreads();
  }

  auto stage = [&](int64_t tile, float* buf) {
    if (tile < tiles.count) {
      int b, x0, y0;
      tiles.at(tile, ROWS, b, x0, y0);
      // Rows of `a` with their halo: 4 cells at once where a row's cells are
      // aligned and all in the grid.
      constexpr int kARows = G::kCin * (ROWS + 2);
      const float* src;
      float* dst;
      auto row = [&](int rr) -> bool {
        const int c = rr / (ROWS + 2), r = rr - c * (ROWS + 2), y = y0 - 1 + r;
        dst = buf + c * G::kAPlane + r * kARow + 4;
        src = a + ((int64_t)b * G::kCin + c) * n + (int64_t)y * W + x0;
        return y >= 0 && y < H;
      };
      if (vec && x0 + 32 <= W) {
        for (int k = tid; k < kARows * 8; k += kTrainThreads) {
          const bool in = row(k >> 3);
          const int q = (k & 7) * 4;
          if (in) cp_async16(dst + q, src + q);
          else *reinterpret_cast<float4*>(dst + q) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
      } else {
        for (int rr = warp; rr < kARows; rr += 4) {
          const bool in = row(rr);
          if (in && x0 + lane < W) cp_async4(dst + lane, src + lane);
          else dst[lane] = 0.0f;
        }
      }
      for (int k = tid; k < kARows * 2; k += kTrainThreads) {
        const bool in = row(k >> 1);
        const int c = k & 1 ? 32 : -1;
        if (in && x0 + c >= 0 && x0 + c < W) cp_async4(dst + c, src + c);
        else dst[c] = 0.0f;
      }
      for (int rr = warp; rr < COUT * ROWS; rr += 4) {
        const int c = rr / ROWS, r = rr - c * ROWS, y = y0 + r;
        float* d = buf + G::kCin * G::kAPlane + r * G::kDRow + lane * G::kDCell + c;
        if (y < H && x0 + lane < W)
          cp_async4(d, dz + ((int64_t)b * COUT + c) * n + (int64_t)y * W + x0 + lane);
        else *d = 0.0f;
      }
    }
    cp_async_commit();
  };

  const int pxs = tid % PXS, cig = tid / PXS % CIG, cog = tid / (PXS * CIG);
  f32x2 acc[TCO / 2][2][9];
  float bsum = 0.0f;  // of channel tid % COUT, columns tid / COUT * 8 + 0..7
  auto sweep = [&](auto guarded) {
#pragma unroll
    for (int k = 0; k < TCO / 2; k++)
#pragma unroll
      for (int c = 0; c < 2; c++)
#pragma unroll
        for (int t = 0; t < 9; t++) acc[k][c][t] = 0;
    int cur = 0;
    stage(blockIdx.x, smem);
    for (int64_t tile = blockIdx.x; tile < tiles.count; tile += gridDim.x, cur ^= 1) {
      stage(tile + gridDim.x, smem + (cur ^ 1) * G::kBuf);
      cp_async_wait_all_but<1>();
      __syncthreads();
      const float* sa = smem + cur * G::kBuf;
      const float* sd = sa + G::kCin * G::kAPlane;
      if constexpr (decltype(guarded)::value) {
        int b, x0, y0;
        tiles.at(tile, ROWS, b, x0, y0);
#pragma unroll 1
        for (int p = 0; p < ROWS / PXS * 32; p++) {
          const int r = pxs + (p >> 5) * PXS, px = p & 31, x = x0 + px, y = y0 + r;
          if (x >= W || y >= H) continue;
#pragma unroll
          for (int k = 0; k < TCO; k++) {
            const float d = sd[r * G::kDRow + px * G::kDCell + cog * TCO + k];
            if (d == 0.0f) continue;
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
              for (int t = 0; t < 9; t++) {
                const int xx = x + t % 3 - 1, yy = y + t / 3 - 1;
                if (xx < 0 || yy < 0 || xx >= W || yy >= H) continue;
                const float v =
                    sa[(cig + c * CIG) * G::kAPlane + (r + t / 3) * kARow + 3 + px + t % 3];
                float s[2];
                unpack2(acc[k / 2][c][t], s[0], s[1]);
                s[k & 1] = fmaf(d, v, s[k & 1]);
                acc[k / 2][c][t] = pack2(s[0], s[1]);
              }
          }
        }
      } else {
#pragma unroll 1
        for (int r = pxs; r < ROWS; r += PXS) {
          const float* pa = sa + cig * G::kAPlane + r * kARow + 3;
          const float* pd = sd + r * G::kDRow + cog * TCO;
#pragma unroll 1
          for (int x = 0; x < 32; x += 4, pa += 4, pd += 4 * G::kDCell) {
            f32x2 d[4][TCO / 2];
#pragma unroll
            for (int j = 0; j < 4; j++) {
              if constexpr (TCO == 4) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(pd + j * G::kDCell);
                d[j][0] = v.x;
                d[j][1] = v.y;
              } else {
                d[j][0] = *reinterpret_cast<const f32x2*>(pd + j * G::kDCell);
              }
            }
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
              for (int dy = 0; dy < 3; dy++) {
                const float* p = pa + c * CIG * G::kAPlane + dy * kARow;
                const float4 v = *reinterpret_cast<const float4*>(p + 1);
                const float e[6] = {p[0], v.x, v.y, v.z, v.w, p[5]};
#pragma unroll
                for (int j = 0; j < 6; j++) {
                  const f32x2 vv = pack2(e[j], e[j]);
#pragma unroll
                  for (int dx = 0; dx < 3; dx++) {  // cell j - dx sees it at its tap dx
                    if (j - dx < 0 || j - dx > 3) continue;
#pragma unroll
                    for (int k = 0; k < TCO / 2; k++)
                      acc[k][c][dy * 3 + dx] = fma2(d[j - dx][k], vv, acc[k][c][dy * 3 + dx]);
                  }
                }
              }
          }
        }
        if (tid < COUT * 4) {
          const float* p = sd + tid / COUT * 8 * G::kDCell + tid % COUT;
#pragma unroll
          for (int r = 0; r < ROWS; r++)
#pragma unroll
            for (int x = 0; x < 8; x += 2)
              bsum += p[r * G::kDRow + x * G::kDCell] + p[r * G::kDRow + (x + 1) * G::kDCell];
        }
      }
      __syncthreads();
    }
  };
  sweep(std::false_type());
  if (tid < COUT * 4) s_bias[tid] = bsum;
  float zero = 0.0f;  // stays 0 while every sum is finite
#pragma unroll
  for (int k = 0; k < TCO / 2; k++)
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int t = 0; t < 9; t++) {
        float lo, hi;
        unpack2(acc[k][c][t], lo, hi);
        zero = fmaf(lo, 0.0f, fmaf(hi, 0.0f, zero));
      }
  if (__syncthreads_or(!(zero == 0.0f))) sweep(std::true_type());

  const bool alone = gridDim.x == 1;
  float* sums = part + (int64_t)blockIdx.x * G::kSums;
#pragma unroll
  for (int k = 0; k < TCO && k < COUT; k++)
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int t = 0; t < 9; t++) {
        float s[2];
        unpack2(acc[k / 2][c][t], s[0], s[1]);
        float v = s[k & 1];
#pragma unroll
        for (int o = 1; o < PXS; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (pxs == 0) {
          const int i = ((cog * TCO + k) * G::kCin + cig + c * CIG) * 9 + t;
          if (alone) gw[i] += v;
          else sums[i] = v;
        }
      }
  if (tid < COUT) {
    const float v = (s_bias[tid] + s_bias[COUT + tid]) + (s_bias[2 * COUT + tid] + s_bias[3 * COUT + tid]);
    if (alone) gb[tid] += v;
    else sums[G::kWeights + tid] = v;
  }
}

// Adds the blocks' sums to the gradients: 32 sums a block, the blocks' parts
// split over 8 warps.
__global__ void __launch_bounds__(256) train_wsum_kernel(const float* __restrict__ part, int blocks,
                                                         int weights, int sums,
                                                         float* __restrict__ gw,
                                                         float* __restrict__ gb) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  float s = 0.0f;
  if (i < sums)
    for (int b = warp; b < blocks; b += 8) s += part[(int64_t)b * sums + i];
  red[warp][lane] = s;
  __syncthreads();
  if (warp || i >= sums) return;
#pragma unroll
  for (int k = 1; k < 8; k++) s += red[k][lane];
  if (i < weights) gw[i] += s;
  else gb[i - weights] += s;
}

// Mean squared error over the cells at least `margin` cells inside each
// grid: dy = 2 (y - t) / count there, 0 elsewhere; loss (sum) accumulated, by
// one addition per block (at most 304 of them, so that their order matters
// little).
__global__ void __launch_bounds__(256) ws_mse_kernel(const float* __restrict__ y,
                                                     const float* __restrict__ t,
                                                     float* __restrict__ dy,
                                                     float* __restrict__ loss, int W, int H, int B,
                                                     int margin, float inv_count) {
  const int64_t n = (int64_t)W * H;
  float l = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n * B; i += (int64_t)gridDim.x * 256) {
    const int64_t c = i % n;
    const int x = (int)(c % W), yy = (int)(c / W);
    const bool in = x >= margin && yy >= margin && x < W - margin && yy < H - margin;
    const float d = y[i] - t[i];
    dy[i] = in ? 2.0f * d * inv_count : 0.0f;
    l += in ? d * d * inv_count : 0.0f;
  }
  __shared__ float red[8];
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < 8; k++) l += red[k];
    if (l != 0.0f) atomicAdd(loss, l);
  }
}

__global__ void ws_adam_kernel(float* __restrict__ p, const float* __restrict__ g,
                               float* __restrict__ m, float* __restrict__ v, int n, float lr,
                               float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

namespace {


// The device's SM count, the kernels' shared memory allowed for.
cageo_status train_sms(int* sms) {
  static PerDevice cache;
  return per_device(cache, sms, [&](int dev, int* v) -> cageo_status {
    auto allow = [](auto fn, size_t bytes) {
      return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    CAGEO_CUDA(allow(train_conv32_kernel<false>, conv32_smem(32)));
    CAGEO_CUDA(allow(train_conv32_kernel<true>, conv32_smem(32)));
    CAGEO_CUDA((allow(train_wgrad_kernel<32, 4, 2, 8, 8>, Wgrad<32, 4, 2, 8, 8>::kSmem)));
    CAGEO_CUDA((allow(train_wgrad_kernel<32, 4, 16, 1, 4>, Wgrad<32, 4, 16, 1, 4>::kSmem)));
    CAGEO_CUDA((allow(train_wgrad_kernel<1, 2, 16, 8, 8>, Wgrad<1, 2, 16, 8, 8>::kSmem)));
    int m = 0;
    CAGEO_CUDA(cudaDeviceGetAttribute(&m, cudaDevAttrMultiProcessorCount, dev));
    *v = std::max(m, 1);
    return CAGEO_OK;
  });
}

struct Shape {
  int W, H, B, sms;
  int64_t cells() const { return (int64_t)W * H * B; }
  // Grids whose rows fill little of a tile's.  Forward, 16 x 12x20000: tiles 5.9
  // ms, a cell a thread 3.9; 64 x 3x400: 0.52 and 0.13; from 14 columns on tiles.
  bool narrow() const { return W <= 12; }
  // The weight gradients' blocks are as many as their sums have room for, 289
  // cells each, which few columns spread over many tiles; a block per channel pair
  // walks all cells alone.  A backward pass of 2 x 3x400: 0.35 ms by tiles, 0.11 by
  // pairs; of 16 x 4x300 0.32 and 0.36; of 64 x 3x400 0.71 and 1.23.
  bool narrow_sums() const { return W <= 24 && cells() * W <= 65536; }
  bool aligned(std::initializer_list<const void*> ptrs) const {
    uintptr_t m = W & 3 ? 1 : 0;
    for (const void* p : ptrs) m |= (uintptr_t)p & 15u;
    return m == 0;
  }
};

template <bool FLIP>
void conv32(const Shape& g, const float* in, int cin, const float* w, const float* bias,
            const float* mask, float* out, int relu, cudaStream_t s) {
  if (g.narrow()) {
    train_conv_narrow_kernel<32, FLIP><<<(unsigned)((g.cells() + kTrainThreads - 1) / kTrainThreads),
                                         kTrainThreads, 32 * cin * 9 * sizeof(float), s>>>(
        in, cin, w, bias, mask, out, g.W, g.H, g.B, relu);
    return;
  }
  const int64_t tiles = TrainTiles(g.W, g.H, g.B, kConvRows).count;
  train_conv32_kernel<FLIP><<<(unsigned)std::min<int64_t>(tiles, 3 * g.sms), kTrainThreads,
                              conv32_smem(cin), s>>>(in, cin, w, bias, mask, out, g.W, g.H, g.B,
                                                     relu, g.aligned({out, mask}));
}

// part: scratch of 32 * W * H * B floats.
template <int COUT, int TCO, int CIG, int PXS, int ROWS>
void wgrad(const Shape& g, const float* dz, const float* a, float* gw, float* gb, float* part,
           cudaStream_t s) {
  using K = Wgrad<COUT, TCO, CIG, PXS, ROWS>;
  if (g.narrow_sums()) {
    train_wgrad_narrow_kernel<<<COUT * K::kCin, 256, 0, s>>>(dz, COUT, a, K::kCin, gw, gb, g.W, g.H,
                                                             g.B);
    return;
  }
  const int64_t tiles = TrainTiles(g.W, g.H, g.B, ROWS).count;
  const int64_t room = 32 * g.cells() / K::kSums;
  const int per = std::min(3, 220 * 1024 / K::kSmem);  // resident blocks per SM
  const int blocks = (int)std::max<int64_t>(1, std::min({tiles, room, (int64_t)per * g.sms}));
  train_wgrad_kernel<COUT, TCO, CIG, PXS, ROWS><<<blocks, kTrainThreads, K::kSmem, s>>>(
      dz, a, gw, gb, part, g.W, g.H, g.B, g.aligned({dz, a}));
  if (blocks > 1)
    train_wsum_kernel<<<(K::kSums + 31) / 32, 256, 0, s>>>(part, blocks, K::kWeights, K::kSums, gw,
                                                          gb);
}

}  // namespace

}  // namespace cageo

using namespace cageo;

extern "C" cageo_status cageo_ws_forward(const float* d_params, const float* d_feat, int W,
                                         int H, int B, float* d_a1, float* d_a2, float* d_out,
                                         cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_params && d_feat && d_a1 && d_a2 && d_out && valid_dims(W, H) && B >= 1,
                  "pointers, size and batch");
  Shape g{W, H, B, 1};
  cageo_status st = train_sms(&g.sms);
  if (st) return st;
  conv32<false>(g, d_feat, 4, d_params + kOffW1, d_params + kOffB1, nullptr, d_a1, 1, stream);
  conv32<false>(g, d_a1, 32, d_params + kOffW2, d_params + kOffB2, nullptr, d_a2, 1, stream);
  if (g.narrow()) {
    train_conv_narrow_kernel<1, false><<<(unsigned)((g.cells() + kTrainThreads - 1) / kTrainThreads),
                                         kTrainThreads, 32 * 9 * sizeof(float), stream>>>(
        d_a2, 32, d_params + kOffW3, d_params + kOffB3, nullptr, d_out, W, H, B, 0);
  } else {
    const int64_t tiles = TrainTiles(W, H, B, kConvRows).count;
    train_conv1_kernel<<<(unsigned)std::min<int64_t>(tiles, 7 * g.sms), kTrainThreads, 0, stream>>>(
        d_a2, d_params + kOffW3, d_params + kOffB3, d_out, W, H, B);
  }
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

extern "C" cageo_status cageo_ws_backward(const float* d_params, const float* d_feat,
                                          const float* d_a1, const float* d_a2,
                                          const float* d_dout, int W, int H, int B,
                                          float* d_grad, float* d_tmp1, float* d_tmp2,
                                          float* d_wflip, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_params && d_feat && d_a1 && d_a2 && d_dout && d_grad && d_tmp1 && d_tmp2 &&
                      d_wflip && valid_dims(W, H) && B >= 1,
                  "pointers, size and batch");
  Shape g{W, H, B, 1};
  cageo_status st = train_sms(&g.sms);
  if (st) return st;
  // Per layer: weight gradients (whose blocks' sums go to the scratch that is
  // free then), and the gradient of its input, masked by its ReLU.
  wgrad<1, 2, 16, 8, 8>(g, d_dout, d_a2, d_grad + kOffW3, d_grad + kOffB3, d_tmp1, stream);
  conv32<true>(g, d_dout, 1, d_params + kOffW3, nullptr, d_a2, d_tmp1, 0, stream);
  wgrad<32, 4, 16, 1, 4>(g, d_tmp1, d_a1, d_grad + kOffW2, d_grad + kOffB2, d_tmp2, stream);
  conv32<true>(g, d_tmp1, 32, d_params + kOffW2, nullptr, d_a1, d_tmp2, 0, stream);
  // (Layer 1's input, the features, needs no gradient.)
  wgrad<32, 4, 2, 8, 8>(g, d_tmp2, d_feat, d_grad + kOffW1, d_grad + kOffB1, d_tmp1, stream);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

extern "C" cageo_status cageo_ws_mse(const float* d_y, const float* d_target, float* d_dy,
                                     float* d_loss, int W, int H, int B, int margin,
                                     cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_y && d_target && d_dy && d_loss && valid_dims(W, H) && B >= 1,
                  "pointers, size and batch");
  CAGEO_CHECK_ARG(margin >= 0 && 2 * margin < W && 2 * margin < H, "margin");
  const int64_t n = (int64_t)W * H * B;
  const float cnt = (float)(W - 2 * margin) * (float)(H - 2 * margin) * (float)B;
  ws_mse_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 304), 256, 0, stream>>>(
      d_y, d_target, d_dy, d_loss, W, H, B, margin, 1.0f / cnt);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}

extern "C" cageo_status cageo_ws_adam(float* d_params, const float* d_grad, float* d_m,
                                      float* d_v, int n, float lr, float beta1, float beta2,
                                      float eps, int step, cudaStream_t stream) {
  CAGEO_CHECK_ARG(d_params && d_grad && d_m && d_v && n > 0 && step >= 1, "arguments");
  const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
  ws_adam_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(d_params, d_grad, d_m, d_v, n, lr,
                                                                  beta1, beta2, eps, c1, c2);
  CAGEO_CUDA(cudaGetLastError());
  return CAGEO_OK;
}
