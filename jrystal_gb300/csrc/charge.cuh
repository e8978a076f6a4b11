// The charge factor of ChargeFix (plan.h).
#pragma once
#include "plan.h"

namespace jrg {

// the charge factor s of ChargeFix (every thread of the block gets it)
__device__ __forceinline__ double charge_scale(const ChargeFix& cf, double* red) {
  if (!cf.qpart) return 1.0;
  double a = 0.0, t = 0.0;
  for (int i = threadIdx.x; i < cf.nq; i += blockDim.x) a += cf.qpart[i];
  for (int i = threadIdx.x; i < cf.nocc; i += blockDim.x) t += cf.occ[i];
  block_sum2(a, t, red);
  a *= cf.dv;
  return (a > 0.0 && t > 0.0) ? t / a : 1.0;
}

}  // namespace jrg
