// The gate's activations, shared by the gate kernels and the chunk preparation (the same values from either).
#pragma once

#include "kda_common.cuh"

namespace kda {

// softplus and its derivative (the sigmoid) from one exponential: log(1 + e^x), e^x / (1 + e^x); identity / 1 above 20.
// Below -15 the sum 1 + e^x would round the small term away: log(1 + e) = e there to fp32 accuracy.
__device__ __forceinline__ float softplusf_(float x, float& sig) {
  const float e = __expf(fminf(x, 20.f));
  const float t = 1.f + e;
  sig = x > 20.f ? 1.f : __fdividef(e, t);
  return x > 20.f ? x : (x < -15.f ? e : __logf(t));
}

// g of the raw gate input x (dt_bias already added), al = exp(A_log[h])
__device__ __forceinline__ float gate_value(float x, float al, int use_lb, float lb) { return use_lb ? lb * sigmoid_fast(al * x) : -al * softplus_fast(x); }

}  // namespace kda
