// The gate network's shape and activation, shared by the inference and training kernels.
#pragma once

#include "kernels.h"

namespace ccnn {

constexpr int kGC = 8;  // channels
// parameter vector: W1 [map][tap], b1, W2 [map][input map][tap], b2, W3 [octave][map], b3
constexpr int kW1 = 0, kB1 = kW1 + kGC * 9, kW2 = kB1 + kGC, kB2 = kW2 + kGC * kGC * 9, kW3 = kB2 + kGC, kB3 = kW3 + kGK * kGC;
static_assert(kB3 + kGK == kGateParams, "gate parameter layout");

__device__ __forceinline__ float lrelu(float z) { return z > 0.f ? z : 0.1f * z; }

}  // namespace ccnn
