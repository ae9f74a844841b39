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

// Exponent (base 2) of the Gaussian at (dx, dy).  Explicit intrinsics: the
// adjoint evaluates the identical sequence.
__device__ __forceinline__ float exponent2(float A, float B, float C, float dx, float dy) {
  const float ax2 = __fmul_rn(__fmul_rn(A, dx), dx);
  const float q = __fmul_rn(B, dx);
  return __fmaf_rn(__fmaf_rn(C, dy, q), dy, ax2);
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

// From the thread's sums (e[0] = sum Gd, e[1] = sum Gd dy, e[2] = sum Gd dy^2
// over its pixels; u = o Gd = dL/dpower) to the gradient terms: e0 =
// dL/dndc_x, e1 = dL/dndc_y, e2..e4 = (sum u dx^2, sum u dx dy, sum u dy^2)
// for the conic (scaled by -1/2, -1, -1/2 at the atomics), e5 = dL/dopacity.
__device__ __forceinline__ void adjoint_finish(float dx, float o, const float4 &s2,
                                               const float4 &s3, float *e) {
  e[5] = e[0];
  const float su = o * e[0], suy = o * e[1], suy2 = o * e[2];
  const float sux = dx * su;
  e[0] = sux * s2.z + suy * s2.w;
  e[1] = suy * s3.x + sux * s3.y;
  e[2] = sux * dx;
  e[3] = suy * dx;
  e[4] = suy2;
}

// Transposed reduce-scatter of the 9 gradient slots over the warp, 12
// shuffles: each level halves the slots a lane keeps (5 | 4, 3 | 2, 2 | 1,
// 1 | 1) and adds its partner's copy of them; afterwards the even lane 2q
// holds the warp sum of slot slot9(q) (q = lane bits 4..1), none when that
// is >= 9.
__device__ __forceinline__ float warp_reduce_scatter9(const float (&v)[9], int lane) {
  float a[5], b[3], c[2];
  {
    const bool hi = lane & 16;
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float up = i < 4 ? v[5 + i] : 0.f;
      a[i] = (hi ? up : v[i]) + __shfl_xor_sync(FULL, hi ? v[i] : up, 16);
    }
  }
  {
    const bool hi = lane & 8;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const float up = i < 2 ? a[3 + i] : 0.f;
      b[i] = (hi ? up : a[i]) + __shfl_xor_sync(FULL, hi ? a[i] : up, 8);
    }
  }
  {
    const bool hi = lane & 4;
    c[0] = (hi ? b[2] : b[0]) + __shfl_xor_sync(FULL, hi ? b[0] : b[2], 4);
    c[1] = (hi ? 0.f : b[1]) + __shfl_xor_sync(FULL, hi ? b[1] : 0.f, 4);
  }
  const bool hi = lane & 2;
  const float d = (hi ? c[1] : c[0]) + __shfl_xor_sync(FULL, hi ? c[0] : c[1], 2);
  return d + __shfl_xor_sync(FULL, d, 1);
}

// slot of the even lane 2q after warp_reduce_scatter9 (15: none)
__device__ __forceinline__ int slot9(int q) {
  return (int)((0xFFF8F765FF43F210ull >> (4 * q)) & 15u);
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
