// Pieces of the velocity-Verlet kernels (k_nve.cu, k_mixed.cu).
#pragma once
#include "internal.h"

namespace cacg {

// dt/(2m) of a type: a select over constant indices, so that the table stays
// in the parameter space (a runtime index into a by-value parameter array
// would copy it to each thread's local memory)
__device__ __forceinline__ double type_scale(const TypeScale &t, int ty) {
  double d = t.v[0];
#pragma unroll
  for (int k = 1; k <= MAXT; k++) d = ty == k ? t.v[k] : d;
  return d;
}

// a + b * c: the reference's multiply-then-add, or one fused multiply-add in
// the FP64 (FMA) and mixed modes (FP64 instructions are scarce on this GPU:
// the integrators are bound by their FP64 issue, not by HBM)
template <bool FUSED>
__device__ __forceinline__ double madd(double a, double b, double c) {
  return FUSED ? fma(b, c, a) : __dadd_rn(a, __dmul_rn(b, c));
}

// the half-steps before a step's positions: one, or two when the previous
// step's second half-step was left to this one (each rounded by itself)
template <bool FUSED, int KICKS>
__device__ __forceinline__ double kick(double v, double s, double f) {
  double w = madd<FUSED>(v, s, f);
  if (KICKS == 2) w = madd<FUSED>(w, s, f);
  return w;
}

}  // namespace cacg
