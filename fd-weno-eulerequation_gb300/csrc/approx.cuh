// The hardware's FP32 approximations as single instructions: relative error at
// most 2^-23 (reciprocal, square root) and 2^-22.9 (reciprocal square root);
// subnormal operands and results count as zero.
#pragma once

namespace wenofd {
namespace dev {

__device__ __forceinline__ float rcp_ftz(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float sqrt_ftz(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

}  // namespace dev
}  // namespace wenofd
