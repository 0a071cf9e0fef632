// front.cuh -- the "front" of a realization: convolved noise -> realistic
// DEM -> stream burning -> pit-fill quantization, fused into the epilogue of
// the convolution kernels.  Shared by noise_conv.cu (kernels) and
// pipeline.cu (launch).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "fillflags.cuh"
#include "stage_math.cuh"

namespace cageo {

// Per-cell static code computed once per pipeline from the stream raster:
//   bits 0-4: index (1..) into the burn-factor table of the nearest stream
//             within the bevel radius, 0 = none;
//   bit 6   : tracing stream   (streams >= 0, FlowTracingAlgorithmCPUOpenMP.h:58)
//   bit 7   : burning stream   (streams != NODATA, StreamBurningAlgorithmCPUOpenMP.h:51)
constexpr uint8_t kCodeTraceStream = 0x40;
constexpr uint8_t kCodeBurnStream = 0x80;
constexpr int kMaxBurnClasses = 31;

// Tile shapes of the fused front's separable convolution (output columns x
// rows per block), chosen per pipeline by its autotuner; the outputs never
// depend on the shape.
constexpr int kConvTiles = 4;

struct FrontParams {
  const float* dem;        // W*H
  const uint8_t* code;     // W*H static codes
  float* q;                // W*H output: quantized burned realistic DEM (grid blockIdx.z of a stack after it)
  unsigned int* min_ord;   // ordered-uint min of q (pit-fill minE), one per grid of a stack
  int* anomaly;            // set when the precomputed burn factor may not apply (per grid of a stack)
  float nodata_dem;
  int quantize;            // 1: the CPU fill's 1 mm quantization; 0: raw (exact fill)
  int quick;               // NODATA does not lie in (0, 4000)
  // The pit fill's seeds: a tile holding an outlet (a border cell or a cell
  // at 0) is marked.
  uint8_t* tseed;          // fill tile seeds (of the whole, possibly stacked, grid)
  int tiles_x;             // fill tiles per row
  int row0;                // this grid's first row in the stacked grid
  int W, H;                // this grid's size (its border)
  float factor[kMaxBurnClasses + 1];  // factor[0] unused
};

// One output of the fused front (column x, row y of this grid) from the
// convolved value and the cell's DEM value and static code: the quantized
// burned elevation.  Flags what the precomputed factors cannot cover.
__device__ __forceinline__ float front_value(const FrontParams& p, float conv, float dem, uint8_t c) {
  float v = realistic_value(dem, conv, p.nodata_dem);
  if (c & kCodeBurnStream) {
    // The reference tests a stream neighbour's elevation against NODATA;
    // the precomputed factors assume that test passes.
    if (v == p.nodata_dem) atomicExch(p.anomaly + blockIdx.z, 1);
    v = 0.0f;
  }
  const int k = c & 0x1f;
  if (k) v = __fmul_rn(v, p.factor[k]);
  return p.quantize ? fill_quantize(v, p.nodata_dem) : v;
}

// Whether the cell is an outlet of the pit fill, and the mark of its tile.
__device__ __forceinline__ bool front_outlet(const FrontParams& p, int x, int y, float q) {
  return q == 0.0f || x == 0 || y == 0 || x == p.W - 1 || y == p.H - 1;
}
__device__ __forceinline__ void front_seed(const FrontParams& p, int x, int y) {
  p.tseed[((p.row0 + (int)blockIdx.z * p.H + y) >> 5) * p.tiles_x + (x >> 5)] = 1;
}

}  // namespace cageo
