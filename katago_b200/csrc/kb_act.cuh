// Activation functions.  The accurate ones are for the fp32 paths; the fast ones, for reduced-precision outputs (fp16 / bf16),
// use special-function-unit approximations whose error is far below the output rounding.
#pragma once

#include "../../include/kb_modelblob.h"

namespace kb {

// Activation functions (eigenbackend.cpp:749-760; MISH_SCALE8 from desc.cpp:402-432).
__device__ __forceinline__ float mishF(float x) {
  // x * tanh(softplus(x)), softplus linear above 20
  float sp = (x > 20.0f) ? x : log1pf(expf(x));
  return x * tanhf(sp);
}
__device__ __forceinline__ float applyActF(float x, int act) {
  switch(act) {
    case KB_ACT_RELU: return fmaxf(x, 0.0f);
    case KB_ACT_MISH: return mishF(x);
    case KB_ACT_SILU: return x / (1.0f + expf(-x));
    case KB_ACT_MISH_SCALE8: {
      float x8 = 8.0f * x;
      float sp = (x8 > 20.0f) ? x8 : log1pf(expf(x8));
      return x * tanhf(sp);
    }
    default: return x;
  }
}

__device__ __forceinline__ float ex2Approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcpApprox(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// mish(x) = x*tanh(softplus(x)) = x - 2x / (n^2 + 2n + 2) with n = e^x (exact identity).  Large x: n = inf, the
// reciprocal is 0 and the result is x; very negative x: n = 0 and the result is 0.  No clamp is needed.
__device__ __forceinline__ float fastMish(float x) {
  const float n = ex2Approx(x * 1.4426950408889634f);
  const float r = rcpApprox(fmaf(n, n + 2.0f, 2.0f));
  return fmaf(-2.0f, x * r, x);
}
__device__ __forceinline__ float fastAct(float x, int act) {
  switch(act) {
    case KB_ACT_RELU: return fmaxf(x, 0.0f);
    case KB_ACT_MISH: return fastMish(x);
    case KB_ACT_SILU: return x * rcpApprox(1.0f + ex2Approx(x * -1.4426950408889634f));
    case KB_ACT_MISH_SCALE8: {
      const float n = ex2Approx(x * (8.0f * 1.4426950408889634f));
      const float r = rcpApprox(fmaf(n, n + 2.0f, 2.0f));
      return fmaf(-2.0f, x * r, x);
    }
    default: return x;
  }
}

}  // namespace kb
