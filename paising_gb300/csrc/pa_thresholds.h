// pa_thresholds.h -- per-temperature acceptance thresholds, shared by the
// host (fixed schedules, computed with the host's exp like the reference) and
// the adaptive-step kernel (schedules chosen on the device, device exp).
#pragma once

#include <cmath>
#include <cstdint>

#include "pa_state.h"

namespace pa {

// Integer thresholds of one temperature (kThrPerStep words):
//   [0..9]  SSC Boltzmann table boltz[idxT0 + 2 idxT1] = min(1, exp(-2 s sum_nn beta))
//           (PAisingSSC.cu:512-516), stored as ceil(2^32 p) - 1: a reference
//           uniform (H+1)/2^32 is below p iff H < ceil(2^32 p) - 1;
//   [10,11] MSC thresholds ceil(2^32 e^-4b), ceil(2^32 e^-8b) (PAisingMSC.cu:674-675),
//           also those of the native SSC sweep.
__host__ __device__ inline uint32_t threshold_word(double beta, int k) {
  if (k < 10) {
    const int i0 = k & 1, i1 = k >> 1;
    double p = exp(-2.0 * (2 * i0 - 1) * (2 * i1 - 4) * beta);
    if (p > 1.0) p = 1.0;
    return (uint32_t)(ceil(4294967296.0 * p) - 1.0);
  }
  const double t = ceil(4294967296.0 * exp((k == 10 ? -4.0 : -8.0) * beta));
  return t >= 4294967295.0 ? 0xFFFFFFFFu : (uint32_t)t;
}

inline void thresholds(double beta, uint32_t* t) {
  for (int k = 0; k < kThrPerStep; ++k) t[k] = threshold_word(beta, k);
}

}  // namespace pa
