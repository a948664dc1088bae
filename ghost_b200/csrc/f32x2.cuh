// f32x2.cuh -- two FP32 operations in one issue slot (sm_100a packed
// arithmetic); each half is rounded like its scalar form.
#pragma once
#include <cuda_runtime.h>

namespace gb {

__device__ __forceinline__ unsigned long long pk(float2 a) { return *reinterpret_cast<unsigned long long *>(&a); }
__device__ __forceinline__ float2 upk(unsigned long long a) { return *reinterpret_cast<float2 *>(&a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
  return upk(r);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
  return upk(r);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)));
  return upk(r);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pk(a)), "l"(pk(b)), "l"(pk(c)));
  return upk(r);
}
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
// c - a b
__device__ __forceinline__ float2 fnma2(float2 a, float2 b, float2 c) {
  return make_float2(fmaf(-a.x, b.x, c.x), fmaf(-a.y, b.y, c.y));
}

// a + conj b and a - conj b.  Two scalar adds: a packed fma with (1, -1) takes
// one issue slot but the FMA pipe twice as long (512^3 X pass of a step: 5235
// us with the fma, 5044 us with the adds).
__device__ __forceinline__ float2 addc2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y - b.y); }
__device__ __forceinline__ float2 subc2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y + b.y); }

// the same names on pairs of doubles
__device__ __forceinline__ double2 add2(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 sub2(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 mul2(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) {
  return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y));
}
__device__ __forceinline__ double2 fnma2(double2 a, double2 b, double2 c) {
  return make_double2(fma(-a.x, b.x, c.x), fma(-a.y, b.y, c.y));
}
__device__ __forceinline__ double2 both(double a) { return make_double2(a, a); }
__device__ __forceinline__ double2 addc2(double2 a, double2 b) { return make_double2(a.x + b.x, a.y - b.y); }
__device__ __forceinline__ double2 subc2(double2 a, double2 b) { return make_double2(a.x - b.x, a.y + b.y); }

}  // namespace gb
