// rcp.cuh -- reciprocal of a sum held as two FP32 numbers.
#pragma once

namespace tmd {

// 1 / (u + lo) to about half an ulp, for normal u whose reciprocal is normal
// too and |lo| of at most an ulp of u: the hardware's approximate reciprocal
// and one Newton-Raphson step with lo in its residual.
__device__ __forceinline__ float rcp_sum(float u, float lo) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(u));
  return fmaf(r, fmaf(-lo, r, fmaf(-u, r, 1.f)), r);
}

}  // namespace tmd
