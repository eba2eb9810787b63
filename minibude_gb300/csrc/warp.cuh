// warp.cuh -- smallest and largest value of a warp's lanes (sm_100 floating-point redux; a NaN gives way
// to a number).
#pragma once

namespace bude {

__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

} // namespace bude
