// learned.cuh -- sizes and parameter layout of the learned warm start's
// network, shared by its training (learned_train.cu) and inference
// (learned.cu).
#pragma once
#include <cuda_bf16.h>
#include "common.cuh"

namespace cageo {

constexpr int kWsCin = 4, kWsCh = 32;
constexpr int kOffW1 = 0, kOffB1 = 1152, kOffW2 = 1184, kOffB2 = 10400, kOffW3 = 10432,
              kOffB3 = 10720, kWsParams = 10721;
static_assert(kOffB1 == kWsCh * kWsCin * 9 && kOffW2 == kOffB1 + kWsCh &&
                  kOffB2 == kOffW2 + kWsCh * kWsCh * 9 && kOffW3 == kOffB2 + kWsCh &&
                  kOffB3 == kOffW3 + kWsCh * 9 && kWsParams == kOffB3 + 1,
              "parameter layout");

__host__ __device__ inline float bf16_round(float x) {
  return __bfloat162float(__float2bfloat16_rn(x));
}

}  // namespace cageo
