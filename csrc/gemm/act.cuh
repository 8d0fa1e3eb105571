// Ungated activations of the expert MLP and their derivatives, shared by the element-wise kernels and the GEMM epilogues.
#pragma once

namespace b200ep {

// kind: 0 gelu (erf form, as torch.nn.functional.gelu), 1 silu, 2 relu.
__device__ __forceinline__ void act_eval(int kind, float x, float* f, float* df) {
  if (kind == 0) {
    const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * __expf(-0.5f * x * x);
    *f = x * cdf;
    *df = cdf + x * pdf;
  } else if (kind == 1) {
    const float sig = 1.f / (1.f + __expf(-x));
    *f = x * sig;
    *df = sig * (1.f + x * (1.f - sig));
  } else {
    *f = x > 0.f ? x : 0.f;
    *df = x > 0.f ? 1.f : 0.f;
  }
}

}  // namespace b200ep
