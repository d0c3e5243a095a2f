// 1 / (1 + e^-x) with one approximate reciprocal (1 ulp; the exponential in front of it is no better).
#pragma once

namespace b200 {

__device__ __forceinline__ float sigmoid_rcp(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(1.f + __expf(-x)));
  return r;
}

}  // namespace b200
