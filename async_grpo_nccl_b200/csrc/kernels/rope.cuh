// Rotary embedding of a pair of columns, the same operations wherever it is applied (so that the fused and the separate kernels
// agree bit for bit).
#pragma once
#include "../launchers.h"

namespace agrpo {

__device__ __forceinline__ void rope_rotate(float& x1, float& x2, float c, float s) {
  const float a = __fmaf_rn(x1, c, -__fmul_rn(x2, s));
  x2 = __fmaf_rn(x1, s, __fmul_rn(x2, c));
  x1 = a;
}

}  // namespace agrpo
