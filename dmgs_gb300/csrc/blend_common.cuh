// blend_common.cuh — constants and arithmetic shared by the blend kernels
// (blend.cu, blend_warp.cu): whatever decides a pixel's value is evaluated by
// the same sequence of roundings in all of them.
#pragma once
#include "kernels.cuh"

namespace dmgs {

namespace {

constexpr float ALPHA_MIN = 1.0f / 255.0f;
constexpr float ALPHA_MAX = 0.99f;
constexpr float T_EPS = 0.0001f;
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LOG2_255 = 7.994353436858858f;
constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The 48-byte record of list entry id; an entry outside the Gaussians (which
// a correct list never holds) reads as a zero-opacity record, whose
// footprint is empty, so no read leaves the geometry state.
__device__ __forceinline__ void load_record(const BlendView &V, uint32_t id, float4 &f0, float4 &f1,
                                            float4 &f2) {
  if (id < V.P) {
    f0 = V.feat[3 * id]; f1 = V.feat[3 * id + 1]; f2 = V.feat[3 * id + 2];
  } else {
    f0 = f1 = f2 = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A group's share (part of parts) of every span, set to zero by its `width`
// threads.
__device__ __forceinline__ void zero_spans(const ZeroSpans &z, unsigned part, unsigned parts,
                                           unsigned thread, unsigned width) {
  for (int k = 0; k < z.n; ++k) {
    const size_t n = z.words[k];
    const size_t chunk = (((n + parts - 1) / parts) + 3) & ~(size_t)3;
    const size_t a = min(n, chunk * part), e = min(n, a + chunk);
    float *p = z.p[k];
    if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {  // a is a multiple of 4 words (or the end)
      const size_t e4 = a + ((e - a) & ~(size_t)3);
      for (size_t i = a + 4 * (size_t)thread; i < e4; i += 4 * (size_t)width)
        *reinterpret_cast<float4 *>(p + i) = make_float4(0.f, 0.f, 0.f, 0.f);
      for (size_t i = e4 + thread; i < e; i += width) p[i] = 0.f;
    } else {
      for (size_t i = a + thread; i < e; i += width) p[i] = 0.f;
    }
  }
}

}  // namespace

}  // namespace dmgs
