// pa_f32x2.cuh -- packed FP32 arithmetic (two floats in a 64-bit register) of
// sm_103a: one issue slot for two operations, each rounded as the scalar one
// is.  The packed instructions run at half the rate of the scalar ones (64
// lanes per clock and SM against 128, measured), so they save issue slots,
// not FP32 pipe time; the compiler folds the broadcast of one float to both
// halves, a swap of the halves and a negation into the operand.
#pragma once
#include <cuda_runtime.h>

namespace pa {

typedef unsigned long long f2;  // two floats: lane a in the low half, lane b in the high half

__device__ __forceinline__ f2 pk(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 dup(float a) { return pk(a, a); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

}  // namespace pa
