// fillflags.cuh -- the pit fill's passability test.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "stage_math.cuh"

namespace cageo {

// fill_passable() of a quantized value q = RN(k / 1000) (k an integer, as
// fill_quantize makes every value the fill sees).  With minE = 0 and
// 0 <= q < 4096, p = RN(1000 q) lies within 0.25 of k: |q - k/1000| is at
// most half an ulp of q (<= 2^-13), so |1000 q - k| <= 0.123, and rounding
// 1000 q (< 2^22) moves it by at most 0.125.  Then toIndex(q) = trunc(p)
// equals k exactly when p >= k = rint(p), and toElev(k) = RN(k / 1000) = q,
// while toElev of any other index differs from q (values 0.001 apart are
// distinct floats below 8192): passable <=> p >= rint(p), no division.
// Other values take the general test.
__device__ __forceinline__ bool passable_quantized(float q, float minE) {
  if (minE == 0.0f && q >= 0.0f && q < 4096.0f) {
    // rint(p) by adding and taking away 2^23 (0 <= p < 2^22).
    const float p = __fmul_rn(1000.0f, q);
    return p >= __fsub_rn(__fadd_rn(p, 8388608.0f), 8388608.0f);
  }
  return fill_passable(q, minE);
}

}  // namespace cageo
