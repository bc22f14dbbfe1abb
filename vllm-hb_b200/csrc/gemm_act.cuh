// Activations that the tensor-core GEMMs apply to their accumulators.
#pragma once

#include "gemm.h"
#include "tc_core.cuh"

namespace hb {

// Standard normal distribution function by formula 7.1.26 of Abramowitz and Stegun, Handbook of
// Mathematical Functions, for erfc (within 1.5e-7 of the exact value), without branches.
__device__ __forceinline__ float normal_cdf(float g) {
  const float a = fabsf(g) * 0.70710678f;
  const float t = __fdividef(1.f, fmaf(0.3275911f, a, 1.f));
  float p = fmaf(1.061405429f, t, -1.453152027f);
  p = fmaf(p, t, 1.421413741f);
  p = fmaf(p, t, -0.284496736f);
  p = fmaf(p, t, 0.254829592f);
  const float half_erfc = 0.5f * p * t * __expf(-a * a);
  return g < 0.f ? half_erfc : 1.f - half_erfc;
}

// An activation without a gate, on 16 outputs: the form is looked up once.
__device__ __forceinline__ void single_16(float (&v)[16], const GatedAct& act) {
  if (act.form == GatedAct::kErf) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float g = fminf(v[j], act.limit);
      v[j] = g * normal_cdf(g);
    }
  } else if (act.form == GatedAct::kTanh) {
    const float k = __fdividef(2.f, act.limit);
#pragma unroll
    for (int j = 0; j < 16; ++j)  // tanh(y) = 1 - 2 / (1 + e^2y)
      v[j] = act.limit - __fdividef(2.f * act.limit, 1.f + __expf(fminf(v[j] * k, 80.f)));
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float g = fminf(v[j], act.limit), z = act.slope * fmaf(act.cubic * g * g, g, g);
      v[j] = z < -80.f ? 0.f : __fdividef(g, 1.f + __expf(-z));
    }
  }
}

// Gated activation of one output element (fast divide and exponential, as silu_f).
template <bool GENERAL>
__device__ __forceinline__ float gated_f(float g, float u, const GatedAct& act) {
  if (!GENERAL) return silu_f(g) * u;
  g = fminf(g, act.limit);
  u = fminf(fmaxf(u, -act.limit), act.limit);
  if (act.form == GatedAct::kErf) return g * normal_cdf(g) * (u + act.shift);
  const float z = act.slope * fmaf(act.cubic * g * g, g, g);
  // far below zero the gate is zero (the fast divide wants a denominator below 2^126)
  return z < -80.f ? 0.f : __fdividef(g, 1.f + __expf(-z)) * (u + act.shift);
}

}  // namespace hb
