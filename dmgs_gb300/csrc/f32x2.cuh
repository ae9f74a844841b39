// f32x2.cuh — two float32 values in one 64-bit register pair: sm_103a issues
// one instruction for both.  Each form rounds as its scalar one, but a vmul that
// feeds a vadd may come out as one fma (measured: the texture's encoding differs
// from __fadd_rn(a, __fmul_rn(w, v)) in the last bit of 43% of its values, its
// error against 64 bits unchanged): write vfma where the rounding matters.
#pragma once

namespace dmgs {

struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2_make(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float vget(F2 x, int i) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
  return i == 0 ? a : b;
}
__device__ __forceinline__ float vget(float x, int) { return x; }
__device__ __forceinline__ F2 vfma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 vmul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 vadd(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }

}  // namespace dmgs
