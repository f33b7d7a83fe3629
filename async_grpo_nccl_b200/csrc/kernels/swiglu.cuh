// Gradient of silu(g) * u, the same operations wherever it is applied (so that the fused and the separate kernels agree bit for
// bit).
#pragma once

namespace agrpo {

__device__ __forceinline__ void swiglu_grad(float g, float u, float d, float& dg, float& du) {
  const float s = 1.f / (1.f + __expf(-g));
  dg = __fmul_rn(__fmul_rn(__fmul_rn(d, u), s), __fmaf_rn(g, 1.f - s, 1.f));
  du = __fmul_rn(__fmul_rn(d, g), s);
}

}  // namespace agrpo
