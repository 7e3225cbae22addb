// tl_mixed.cuh -- what the FP32 sweeps (tl_mixed.cu) and the FP32 on-chip loop (tl_persist.cu) of
// the precision form share.
#pragma once

#include "tl_kernels.cuh"

namespace tl {

// ---- error-free transformations (Knuth's TwoSum; TwoProduct with FMA) ----
struct Dot2 {
  float s = 0.f, c = 0.f;  // running sum and accumulated error terms
  __device__ __forceinline__ void add(float a, float b) {
    const float p = a * b;
    const float pe = fmaf(a, b, -p);  // a*b = p + pe exactly
    const float t = s + p;
    const float z = t - s;
    const float se = (s - (t - z)) + (p - z);  // s + p = t + se exactly
    s = t;
    c += pe + se;
  }
  __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

__device__ __forceinline__ void mix_finish(MixState* ms) {
  ms->n += 1;
  if (ms->switch_rr > 0.0 && ms->n >= ms->presteps && ms->rr <= ms->switch_rr) {
    ms->status = STOP_SWITCH;
    return;
  }
  // hand over to the host for a residual replacement (the recursive residual fell by delta,
  // or this phase used up its step budget), or stop at the overall cap
  if (!(ms->rr > ms->delta2 * ms->rr_max) || ms->n > ms->max_n || ms->n >= ms->phase_end)
    ms->status = EXIT_CONVERGED;
}

}  // namespace tl
