// Element-wise update rules of the fused optimisers (Adam, AdamW, SGD, ADOPT), shared by the optimiser sweeps and by
// the scoring kernel, which applies them to an entity tile as soon as that tile's gradient is complete.
#pragma once
#include <cuda_runtime.h>

namespace dice {

// The moments are touched once per step: first to leave L2, so that the weights (and gradients) the rest of the step reads
// stay there.
__device__ __forceinline__ float4 ld4_once(const float* p) { return __ldcs(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void st4_once(float* p, float4 v) { __stcs(reinterpret_cast<float4*>(p), v); }

// Step-dependent constants: bias corrections of Adam / AdamW, clip bound of ADOPT; t = number of this step (1-based).
struct OptStepConsts {
  float inv_bc1, inv_sqrt_bc2, clip;
  bool first_step;
};
__device__ __forceinline__ OptStepConsts opt_step_consts(int kind, long long t, float beta1, float beta2) {
  OptStepConsts c;
  c.inv_bc1 = 1.f;
  c.inv_sqrt_bc2 = 1.f;
  if (kind <= 1) {
    c.inv_bc1 = 1.f / (1.f - exp2f(static_cast<float>(t) * log2f(beta1)));
    c.inv_sqrt_bc2 = rsqrtf(1.f - exp2f(static_cast<float>(t) * log2f(beta2)));
  }
  c.clip = sqrtf(sqrtf(static_cast<float>(t - 1)));  // ADOPT: clip bound step^(1/4)
  c.first_step = (t == 1);
  return c;
}

// Square root and quotient for the sweeps: the hardware's approximation and one Newton step on the residual, which an FMA
// gives exactly (P. Markstein, IA-64 and Elementary Functions, 2000).  Within one unit in the last place of the rounded result
// over the normal range (tested against it), without the out-of-line paths of the general operators, whose calls held 60
// registers and with them half of the resident warps of a sweep.
__device__ __forceinline__ float opt_sqrt(float v) {
  float y;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(v));
  const float s = v * y;
  const float r = fmaf(fmaf(-s, s, v), 0.5f * y, s);
  return v == 0.f || v == __int_as_float(0x7f800000) ? v : r;
}
__device__ __forceinline__ float opt_div(float a, float b) {
  float r0;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r0) : "f"(b));
  const float r = fmaf(fmaf(-b, r0, 1.f), r0, r0);
  const float q = a * r;
  const float res = fmaf(fmaf(-b, q, a), r, q);
  if (r0 == 0.f || fabsf(r0) == __int_as_float(0x7f800000)) return a * r0;   // b infinite or zero
  return fabsf(q) == __int_as_float(0x7f800000) ? q : res;                    // overflow: the residual is not a number
}

// One parameter element: returns the updated weight; m / v are updated in place (registers).
__device__ __forceinline__ float opt_update(int kind, float w, float g, float& m, float& v, float lr, float beta1,
                                            float beta2, float eps, float wd, float inv_bc1, float inv_sqrt_bc2,
                                            float clip, bool first_step) {
  if (kind == 0) {
    g = fmaf(wd, w, g);
    m = fmaf(beta1, m, (1.f - beta1) * g);
    v = fmaf(beta2, v, (1.f - beta2) * g * g);
    return w - opt_div(lr * inv_bc1 * m, fmaf(opt_sqrt(v), inv_sqrt_bc2, eps));
  } else if (kind == 1) {
    w *= 1.f - lr * wd;
    m = fmaf(beta1, m, (1.f - beta1) * g);
    v = fmaf(beta2, v, (1.f - beta2) * g * g);
    return w - opt_div(lr * inv_bc1 * m, fmaf(opt_sqrt(v), inv_sqrt_bc2, eps));
  } else if (kind == 2) {
    g = fmaf(wd, w, g);
    return w - lr * g;
  }
  g = fmaf(wd, w, g);  // ADOPT
  if (first_step) {
    v = g * g;
    return w;
  }
  float ng = opt_div(g, fmaxf(opt_sqrt(v), eps));
  ng = fminf(fmaxf(ng, -clip), clip);
  m = m + (1.f - beta1) * (ng - m);
  v = fmaf(beta2, v, (1.f - beta2) * g * g);
  return w - lr * m;
}

}  // namespace dice
