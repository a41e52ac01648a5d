// What the element kernels share: the constants of the local iteration
// (src/fem/IncompatibleModes.hpp:98-127), 3 x 3 algebra and the group sum.
#pragma once

#include <cuda_runtime.h>

namespace sbk {

constexpr int kMaxLocal = 25;
constexpr double kFullStepReduction = 1.0 - 1.0e-4;
constexpr int kMaxLineSearch = 8;
constexpr double kLineSearchRatio = 0.5;
constexpr double kLocalShift = 1.0e-3;
constexpr double kLocalMarquardt = 1.0e-6;
constexpr double kLocalTolerance = 1.0e-8;
constexpr double kLocalRoundOff = 1.0e-13;

__device__ __forceinline__ double det3(const double m[9]) {
  return m[0] * (m[4] * m[8] - m[7] * m[5]) - m[3] * (m[1] * m[8] - m[7] * m[2]) +
         m[6] * (m[1] * m[5] - m[4] * m[2]);
}
__device__ __forceinline__ void inv3(const double m[9], double out[9]) {
  out[0] = m[4] * m[8] - m[5] * m[7];
  out[3] = m[5] * m[6] - m[3] * m[8];
  out[6] = m[3] * m[7] - m[4] * m[6];
  const double det = m[0] * out[0] + m[1] * out[3] + m[2] * out[6];
  const double inv = 1.0 / det;
  out[1] = m[2] * m[7] - m[1] * m[8];
  out[4] = m[0] * m[8] - m[2] * m[6];
  out[7] = m[1] * m[6] - m[0] * m[7];
  out[2] = m[1] * m[5] - m[2] * m[4];
  out[5] = m[2] * m[3] - m[0] * m[5];
  out[8] = m[0] * m[4] - m[1] * m[3];
#pragma unroll
  for (int i = 0; i < 9; ++i) out[i] *= inv;
}

// Reduce-scatter of G values over the G lanes of a group: lane l returns the
// group sum of v[l]. Fixed pairing, so the result is deterministic.
template <int G>
__device__ __forceinline__ double reduce_scatter(double (&v)[G], int lane, unsigned mask) {
  double cur[G];
#pragma unroll
  for (int i = 0; i < G; ++i) cur[i] = v[i];
#pragma unroll
  for (int half = G / 2; half >= 1; half >>= 1) {
    const bool upper = (lane & half) != 0;
#pragma unroll
    for (int j = 0; j < half; ++j) {
      const double send = upper ? cur[j] : cur[half + j];
      const double keep = upper ? cur[half + j] : cur[j];
      cur[j] = keep + __shfl_xor_sync(mask, send, half, G);
    }
  }
  return cur[0];
}

}  // namespace sbk
