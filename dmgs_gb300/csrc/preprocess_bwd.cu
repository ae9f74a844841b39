// preprocess_bwd.cu — per-Gaussian adjoint of the forward geometry.
//
// Input: the per-Gaussian 2D gradients the blend adjoint accumulated
// (dL/d NDC mean, dL/d conic (a, b, c) with b the off-diagonal scalar,
// dL/d opacity, dL/d rgb).  Output: gradients w.r.t. every forward input.
//
// Chain (derived here, conventions of the reference adjoint):
//   conic = inverse(cov2D)           -> dL/dA, dL/dB, dL/dC (cov2D = [[A,B],[B,C]])
//   cov2D = T Sigma T^T, T = J W     -> dL/dSigma = T^T Gs T, dL/dT = 2 Gs T Sigma
//   J(t), t = W m + t0               -> dL/dt with the 1.3 tan(fov) clamp: zero
//                                        gradient through a clamped coordinate,
//                                        the clamped value held constant
//   ndc = hom.xy / (hom.w + 1e-7)    -> dL/dm
//   rgb = max(0, SH(dir) + 0.5)      -> dL/dsh, dL/dm through dir = unit(m - campos)
//   Sigma = (R S)(R S)^T             -> dL/dscale, dL/dquaternion (unnormalised)
// Culled Gaussians (radius 0, empty rectangle in the geometry state) get
// zeros in every output.
#include <algorithm>

#include "kernels.cuh"

namespace dmgs {

namespace {

constexpr int BWD_BLOCK = 128;

// Calls term(k, b_k, db_k/dx, db_k/dy, db_k/dz) for every SH basis function
// of degree <= D at the unit direction (x, y, z) (the real SH basis with the
// PlenOctree constants of utils/sh_utils.py:25-110), k in coefficient order.
template <typename F>
__device__ __forceinline__ void for_each_sh_term(int D, float x, float y, float z, F &&term) {
  term(0, kSH_C0, 0.f, 0.f, 0.f);
  if (D > 0) {
    term(1, -kSH_C1 * y, 0.f, -kSH_C1, 0.f);
    term(2, kSH_C1 * z, 0.f, 0.f, kSH_C1);
    term(3, -kSH_C1 * x, -kSH_C1, 0.f, 0.f);
    if (D > 1) {
      const float xx = x * x, yy = y * y, zz = z * z;
      term(4, kSH_C2[0] * x * y, kSH_C2[0] * y, kSH_C2[0] * x, 0.f);
      term(5, kSH_C2[1] * y * z, 0.f, kSH_C2[1] * z, kSH_C2[1] * y);
      term(6, kSH_C2[2] * (2.f * zz - xx - yy), -2.f * kSH_C2[2] * x, -2.f * kSH_C2[2] * y, 4.f * kSH_C2[2] * z);
      term(7, kSH_C2[3] * x * z, kSH_C2[3] * z, 0.f, kSH_C2[3] * x);
      term(8, kSH_C2[4] * (xx - yy), 2.f * kSH_C2[4] * x, -2.f * kSH_C2[4] * y, 0.f);
      if (D > 2) {
        term(9, kSH_C3[0] * y * (3.f * xx - yy), 6.f * kSH_C3[0] * x * y, kSH_C3[0] * (3.f * xx - 3.f * yy), 0.f);
        term(10, kSH_C3[1] * x * y * z, kSH_C3[1] * y * z, kSH_C3[1] * x * z, kSH_C3[1] * x * y);
        term(11, kSH_C3[2] * y * (4.f * zz - xx - yy), -2.f * kSH_C3[2] * x * y,
             kSH_C3[2] * (4.f * zz - xx - 3.f * yy), 8.f * kSH_C3[2] * y * z);
        term(12, kSH_C3[3] * z * (2.f * zz - 3.f * xx - 3.f * yy), -6.f * kSH_C3[3] * x * z,
             -6.f * kSH_C3[3] * y * z, kSH_C3[3] * (6.f * zz - 3.f * xx - 3.f * yy));
        term(13, kSH_C3[4] * x * (4.f * zz - xx - yy), kSH_C3[4] * (4.f * zz - 3.f * xx - yy),
             -2.f * kSH_C3[4] * x * y, 8.f * kSH_C3[4] * x * z);
        term(14, kSH_C3[5] * z * (xx - yy), 2.f * kSH_C3[5] * x * z, -2.f * kSH_C3[5] * y * z,
             kSH_C3[5] * (xx - yy));
        term(15, kSH_C3[6] * x * (xx - 3.f * yy), kSH_C3[6] * (3.f * xx - 3.f * yy),
             -6.f * kSH_C3[6] * x * y, 0.f);
      }
    }
  }
}

// Geometric adjoint of one (Gaussian, view) pair: every gradient but the SH
// colour's, handed to sink (color, opacity, cov, scale, rot: element index
// and value); the mean's gradient is returned in dm, where the caller adds
// the SH direction term, and the colour's in drgb.
template <typename Sink>
__device__ __forceinline__ void
preprocess_bwd_one(int idx, const ViewParams &vp, const float *__restrict__ viewm_g,
                   const float *__restrict__ projm_g, const float *__restrict__ means,
                   const float *__restrict__ scales, const float *__restrict__ rots,
                   const float *__restrict__ cov3D, const float *__restrict__ gacc,
                   const DmgsGrads &out, const Sink &sink, float (&dm)[3], float (&drgb)[3]) {
  const float4 ga = reinterpret_cast<const float4 *>(gacc)[3 * idx];
  const float4 gb = reinterpret_cast<const float4 *>(gacc)[3 * idx + 1];
  const float gblue = gacc[12 * idx + 8];
  const float dndc_x = ga.x, dndc_y = ga.y;
  const float dca = ga.z, dcb = ga.w, dcc = gb.x;
  const float dop = gb.y;
  drgb[0] = gb.z; drgb[1] = gb.w; drgb[2] = gblue;

  sink.mean2d(dndc_x, dndc_y);
  if (out.dL_dopacity) sink.opacity(dop);
  if (out.dL_dcolors) { sink.color(0, drgb[0]); sink.color(1, drgb[1]); sink.color(2, drgb[2]); }

  float V[16], Pm[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) { V[i] = viewm_g[i]; Pm[i] = projm_g[i]; }  // global or shared
  const float mx = means[3 * idx], my = means[3 * idx + 1], mz = means[3 * idx + 2];

  // --- recompute the forward quantities ---------------------------------
  const float tx0 = V[0] * mx + V[4] * my + V[8] * mz + V[12];
  const float ty0 = V[1] * mx + V[5] * my + V[9] * mz + V[13];
  const float tz = V[2] * mx + V[6] * my + V[10] * mz + V[14];

  float S[6];
  float R[9], sc[3];
  const bool from_sr = (cov3D == nullptr);
  float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (!from_sr) {
#pragma unroll
    for (int i = 0; i < 6; ++i) S[i] = cov3D[6 * idx + i];
  } else {
    q = reinterpret_cast<const float4 *>(rots)[idx];
    const float r = q.x, x = q.y, y = q.z, z = q.w;
    R[0] = 1.f - 2.f * (y * y + z * z); R[1] = 2.f * (x * y - r * z); R[2] = 2.f * (x * z + r * y);
    R[3] = 2.f * (x * y + r * z); R[4] = 1.f - 2.f * (x * x + z * z); R[5] = 2.f * (y * z - r * x);
    R[6] = 2.f * (x * z - r * y); R[7] = 2.f * (y * z + r * x); R[8] = 1.f - 2.f * (x * x + y * y);
    sc[0] = vp.scale_modifier * scales[3 * idx];
    sc[1] = vp.scale_modifier * scales[3 * idx + 1];
    sc[2] = vp.scale_modifier * scales[3 * idx + 2];
    float Mm[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Mm[i * 3 + j] = R[i * 3 + j] * sc[j];
    auto sig = [&](int i, int k) {
      return Mm[i * 3] * Mm[k * 3] + Mm[i * 3 + 1] * Mm[k * 3 + 1] + Mm[i * 3 + 2] * Mm[k * 3 + 2];
    };
    S[0] = sig(0, 0); S[1] = sig(0, 1); S[2] = sig(0, 2); S[3] = sig(1, 1); S[4] = sig(1, 2); S[5] = sig(2, 2);
  }
  const float Sg[9] = {S[0], S[1], S[2], S[1], S[3], S[4], S[2], S[4], S[5]};

  const float limx = 1.3f * vp.tanfovx, limy = 1.3f * vp.tanfovy;
  const float txtz = tx0 / tz, tytz = ty0 / tz;
  const float tx = fminf(limx, fmaxf(-limx, txtz)) * tz;
  const float ty = fminf(limy, fmaxf(-limy, tytz)) * tz;
  const float xmul = (txtz < -limx || txtz > limx) ? 0.f : 1.f;
  const float ymul = (tytz < -limy || tytz > limy) ? 0.f : 1.f;
  const float inv = 1.f / tz, inv2 = inv * inv, inv3 = inv2 * inv;
  const float J00 = vp.fx * inv, J02 = -vp.fx * tx * inv2;
  const float J11 = vp.fy * inv, J12 = -vp.fy * ty * inv2;
  // W_ij = V[i + 4j]
  float T[2][3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    T[0][j] = J00 * V[4 * j + 0] + J02 * V[4 * j + 2];
    T[1][j] = J11 * V[4 * j + 1] + J12 * V[4 * j + 2];
  }
  float TS[2][3];  // T Sigma
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      TS[a][j] = T[a][0] * Sg[j] + T[a][1] * Sg[3 + j] + T[a][2] * Sg[6 + j];
  const float A = TS[0][0] * T[0][0] + TS[0][1] * T[0][1] + TS[0][2] * T[0][2] + 0.3f;
  const float Bc = TS[0][0] * T[1][0] + TS[0][1] * T[1][1] + TS[0][2] * T[1][2];
  const float C = TS[1][0] * T[1][0] + TS[1][1] * T[1][1] + TS[1][2] * T[1][2] + 0.3f;

  // --- conic -> cov2D ----------------------------------------------------
  const float det = A * C - Bc * Bc;
  const float det2 = det * det;
  float dA = 0.f, dB = 0.f, dC = 0.f;
  if (det2 != 0.f) {
    const float id2 = 1.f / det2;
    dA = id2 * (-C * C * dca + Bc * C * dcb - Bc * Bc * dcc);
    dB = id2 * (2.f * Bc * C * dca - (A * C + Bc * Bc) * dcb + 2.f * A * Bc * dcc);
    dC = id2 * (-Bc * Bc * dca + A * Bc * dcb - A * A * dcc);
  }
  // Gs = [[dA, dB/2], [dB/2, dC]]
  const float Gs00 = dA, Gs01 = 0.5f * dB, Gs11 = dC;

  // dL/dSigma_sym = T^T Gs T
  float GT[2][3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    GT[0][j] = Gs00 * T[0][j] + Gs01 * T[1][j];
    GT[1][j] = Gs01 * T[0][j] + Gs11 * T[1][j];
  }
  float dS[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) dS[i * 3 + j] = T[0][i] * GT[0][j] + T[1][i] * GT[1][j];
  if (out.dL_dcov3D) {
    sink.cov(0, dS[0]); sink.cov(1, 2.f * dS[1]); sink.cov(2, 2.f * dS[2]);
    sink.cov(3, dS[4]); sink.cov(4, 2.f * dS[5]); sink.cov(5, dS[8]);
  }

  // dL/dT = 2 Gs T Sigma
  float dT[2][3];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    dT[0][j] = 2.f * (Gs00 * TS[0][j] + Gs01 * TS[1][j]);
    dT[1][j] = 2.f * (Gs01 * TS[0][j] + Gs11 * TS[1][j]);
  }
  // dL/dJ = dL/dT W^T  (W_bk = V[b + 4k])
  float dJ00 = 0.f, dJ02 = 0.f, dJ11 = 0.f, dJ12 = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    dJ00 += dT[0][k] * V[4 * k + 0];
    dJ02 += dT[0][k] * V[4 * k + 2];
    dJ11 += dT[1][k] * V[4 * k + 1];
    dJ12 += dT[1][k] * V[4 * k + 2];
  }
  const float dtx = xmul * (-vp.fx * inv2) * dJ02;
  const float dty = ymul * (-vp.fy * inv2) * dJ12;
  const float dtz = -vp.fx * inv2 * dJ00 - vp.fy * inv2 * dJ11 +
                    2.f * vp.fx * tx * inv3 * dJ02 + 2.f * vp.fy * ty * inv3 * dJ12;
#pragma unroll
  for (int k = 0; k < 3; ++k) dm[k] = V[4 * k] * dtx + V[4 * k + 1] * dty + V[4 * k + 2] * dtz;

  // --- projected mean ----------------------------------------------------
  {
    const float hx = Pm[0] * mx + Pm[4] * my + Pm[8] * mz + Pm[12];
    const float hy = Pm[1] * mx + Pm[5] * my + Pm[9] * mz + Pm[13];
    const float hw = Pm[3] * mx + Pm[7] * my + Pm[11] * mz + Pm[15];
    const float mw = 1.f / (hw + 1e-7f);
    const float mw2 = mw * mw;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float jx = Pm[4 * k] * mw - hx * mw2 * Pm[4 * k + 3];
      const float jy = Pm[4 * k + 1] * mw - hy * mw2 * Pm[4 * k + 3];
      dm[k] += dndc_x * jx + dndc_y * jy;
    }
  }

  // --- scale / rotation --------------------------------------------------
  if (from_sr && (out.dL_dscales || out.dL_drotations)) {
    // dL/dM = 2 dS M,  M = R diag(sc)
    float Mm[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) Mm[i * 3 + j] = R[i * 3 + j] * sc[j];
    float dM[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        dM[i * 3 + j] = 2.f * (dS[i * 3] * Mm[j] + dS[i * 3 + 1] * Mm[3 + j] + dS[i * 3 + 2] * Mm[6 + j]);
    if (out.dL_dscales) {
#pragma unroll
      for (int j = 0; j < 3; ++j)
        sink.scale(j, vp.scale_modifier * (dM[j] * R[j] + dM[3 + j] * R[3 + j] + dM[6 + j] * R[6 + j]));
    }
    if (out.dL_drotations) {
      float G[9];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) G[i * 3 + j] = dM[i * 3 + j] * sc[j];
      const float r = q.x, x = q.y, y = q.z, z = q.w;
      const float dr = 2.f * (-z * G[1] + y * G[2] + z * G[3] - x * G[5] - y * G[6] + x * G[7]);
      const float dx = 2.f * (y * G[1] + z * G[2] + y * G[3] - 2.f * x * G[4] - r * G[5] + z * G[6] +
                              r * G[7] - 2.f * x * G[8]);
      const float dy = 2.f * (-2.f * y * G[0] + x * G[1] + r * G[2] + x * G[3] + z * G[5] - r * G[6] +
                              z * G[7] - 2.f * y * G[8]);
      const float dz = 2.f * (-2.f * z * G[0] - r * G[1] + x * G[2] + r * G[3] - 2.f * z * G[4] +
                              y * G[5] + x * G[6] + y * G[7]);
      sink.rot(dr, dx, dy, dz);
    }
  }
}


// SH adjoint of one view at mean (mx, my, mz): put(j, v) receives element j
// of dL/dsh (3 per coefficient), sh(j) reads the input's; the direction's
// term is added to the mean gradient dm.  drgb is the gradient of the colour
// before its clamp at zero.
template <typename Read, typename Put>
__device__ __forceinline__ void sh_bwd(int D, float mx, float my, float mz, const float *cam,
                                       const float (&drgb)[3], Read &&sh, Put &&put, float (&dm)[3]) {
  const float vx_ = mx - cam[0], vy_ = my - cam[1], vz_ = mz - cam[2];
  const float len = sqrtf(vx_ * vx_ + vy_ * vy_ + vz_ * vz_);
  const float il = 1.f / len;
  const float x = vx_ * il, y = vy_ * il, z = vz_ * il;
  float gdx = 0.f, gdy = 0.f, gdz = 0.f;
  for_each_sh_term(D, x, y, z, [&](int k, float b, float bx, float by, float bz) {
    const float s0 = sh(3 * k), s1 = sh(3 * k + 1), s2 = sh(3 * k + 2);
    put(3 * k, b * drgb[0]);  // may overwrite what sh() reads
    put(3 * k + 1, b * drgb[1]);
    put(3 * k + 2, b * drgb[2]);
    const float dot = s0 * drgb[0] + s1 * drgb[1] + s2 * drgb[2];
    gdx += bx * dot; gdy += by * dot; gdz += bz * dot;
  });
  // d unit(v)/dv . g = (g - u (u . g)) / |v|
  const float ug = x * gdx + y * gdy + z * gdz;
  dm[0] += (gdx - x * ug) * il;
  dm[1] += (gdy - y * ug) * il;
  dm[2] += (gdz - z * ug) * il;
}

__device__ __forceinline__ void apply_clamp(uint32_t flags, float (&drgb)[3]) {
  if (flags & 1) drgb[0] = 0.f;
  if (flags & 2) drgb[1] = 0.f;
  if (flags & 4) drgb[2] = 0.f;
}

// Single-view adjoint, one thread per visible Gaussian of the
// (index-ordered) visible list; the outputs are zero already (the blend adjoint cleared them while
// it ran).  Only ~5-20% of a large scene's Gaussians are visible in a view,
// so a thread per Gaussian ran the ~1,500 instructions of the chain in warps
// of which two lanes in thirty-two had work, and wrote the zeros of the rest
// itself: 273 us at 3M Gaussians (0.14M visible), bound by issue.  Dense
// lanes leave the gathers and the rows written (600 B per visible Gaussian).
// The SH rows are staged per warp in shared memory so that each row's 192
// bytes go out as whole sectors.
constexpr int SHP = 49;  // staging row pitch in floats: lanes writing element j hit different banks

struct RowSink {
  float *m2_, *col_, *op_, *cov_, *sc_, *rot_;  // this Gaussian's row of each output (or null)
  __device__ __forceinline__ void mean2d(float x, float y) const { if (m2_) { m2_[0] = x; m2_[1] = y; } }
  __device__ __forceinline__ void opacity(float v) const { *op_ = v; }
  __device__ __forceinline__ void color(int k, float v) const { col_[k] = v; }
  __device__ __forceinline__ void cov(int k, float v) const { cov_[k] = v; }
  __device__ __forceinline__ void scale(int k, float v) const { sc_[k] = v; }
  __device__ __forceinline__ void rot(float r, float x, float y, float z) const {
    *reinterpret_cast<float4 *>(rot_) = make_float4(r, x, y, z);
  }
};

__global__ void __launch_bounds__(BWD_BLOCK, 5)
preprocess_bwd_list_kernel(ViewParams vp, const float *__restrict__ viewm_g,
                           const float *__restrict__ projm_g, const float *__restrict__ campos_g,
                           int P, int M, const float *__restrict__ means,
                           const float *__restrict__ shs, const float *__restrict__ scales,
                           const float *__restrict__ rots, const float *__restrict__ cov3D,
                           const uint8_t *__restrict__ flags, const float *__restrict__ gacc,
                           const uint32_t *__restrict__ vlist, const uint32_t *__restrict__ counters,
                           DmgsGrads out) {
  extern __shared__ float sm[];
  const int lane = threadIdx.x & 31;
  float *st = sm + (threadIdx.x >> 5) * (32 * SHP);
  const uint32_t V = min(counters[CI_V], (uint32_t)P);
  const int nsh3 = 3 * (vp.D + 1) * (vp.D + 1);
  const int n4 = (nsh3 + 3) / 4;  // float4s of a staged row
  const bool want_dsh = shs != nullptr && out.dL_dsh != nullptr;
  const bool vec_in = (M & 3) == 0 && (reinterpret_cast<uintptr_t>(shs) & 15) == 0;
  const bool vec_out = (M & 3) == 0 && (reinterpret_cast<uintptr_t>(out.dL_dsh) & 15) == 0;
  auto row = [](float *base, int n, size_t i) { return base ? base + n * i : nullptr; };
  for (uint32_t s0 = blockIdx.x * BWD_BLOCK + (threadIdx.x & ~31); s0 < V; s0 += gridDim.x * BWD_BLOCK) {
    const uint32_t s = s0 + lane;
    uint32_t id = s < V ? vlist[s] : 0xffffffffu;
    if (id >= (uint32_t)P) id = 0xffffffffu;
    if (shs != nullptr) {  // the group's SH rows into the staging rows, whole sectors at a time
      if (vec_in) {
        for (int q = lane; q < 32 * n4; q += 32) {
          const int r = q / n4, c = q - r * n4;
          const uint32_t rid = __shfl_sync(0xffffffffu, id, r);
          if (rid == 0xffffffffu) continue;
          const float4 v = __ldg(reinterpret_cast<const float4 *>(shs + (size_t)rid * M * 3) + c);
          float *e = st + r * SHP + 4 * c;
          e[0] = v.x; e[1] = v.y; e[2] = v.z; e[3] = v.w;
        }
      } else {
        for (int q = lane; q < 32 * nsh3; q += 32) {
          const int r = q / nsh3, c = q - r * nsh3;
          const uint32_t rid = __shfl_sync(0xffffffffu, id, r);
          if (rid != 0xffffffffu) st[r * SHP + c] = __ldg(shs + (size_t)rid * M * 3 + c);
        }
      }
    }
    __syncwarp();
    if (id != 0xffffffffu) {
      const size_t i = id;
      RowSink sink;
      sink.m2_ = row(out.dL_dmeans2D, 3, i);
      sink.col_ = row(out.dL_dcolors, 3, i);
      sink.op_ = row(out.dL_dopacity, 1, i);
      sink.cov_ = row(out.dL_dcov3D, 6, i);
      sink.sc_ = row(out.dL_dscales, 3, i);
      sink.rot_ = row(out.dL_drotations, 4, i);
      float dm[3], drgb[3];
      preprocess_bwd_one((int)id, vp, viewm_g, projm_g, means, scales, rots, cov3D, gacc, out, sink, dm, drgb);
      if (shs != nullptr) {
        apply_clamp(flags[id], drgb);
        sh_bwd(vp.D, means[3 * i], means[3 * i + 1], means[3 * i + 2], campos_g, drgb,
               [&](int j) { return st[lane * SHP + j]; },
               [&](int j, float v) { st[lane * SHP + j] = v; }, dm);
      }
      if (out.dL_dmeans3D) {
        float *d = out.dL_dmeans3D + 3 * i;
        d[0] = dm[0]; d[1] = dm[1]; d[2] = dm[2];
      }
    }
    if (!want_dsh) {  // block-uniform
      __syncwarp();
      continue;
    }
    if (id != 0xffffffffu)
      for (int j = nsh3; j < 4 * n4; ++j) st[lane * SHP + j] = 0.f;
    __syncwarp();
    if (vec_out) {
      for (int q = lane; q < 32 * n4; q += 32) {
        const int r = q / n4, c = q - r * n4;
        const uint32_t rid = __shfl_sync(0xffffffffu, id, r);
        const float *e = st + r * SHP + 4 * c;
        if (rid != 0xffffffffu)
          reinterpret_cast<float4 *>(out.dL_dsh + (size_t)rid * M * 3)[c] = make_float4(e[0], e[1], e[2], e[3]);
      }
    } else {
      for (int q = lane; q < 32 * nsh3; q += 32) {
        const int r = q / nsh3, c = q - r * nsh3;
        const uint32_t rid = __shfl_sync(0xffffffffu, id, r);
        if (rid != 0xffffffffu) out.dL_dsh[(size_t)rid * M * 3 + c] = st[r * SHP + c];
      }
    }
    __syncwarp();  // the staged rows are overwritten by the next group
  }
}

// Multi-view adjoint: the gradients of all views of a batch, summed.  A
// Gaussian is visible in few of the views, so a thread per Gaussian looping
// over the views would leave most lanes idle for the geometric part (the
// longest).  Instead the block lists its (Gaussian, view) pairs — thread t's
// Gaussian contributes one pair per view it is visible in, placed by a
// block-wide scan — and the threads take the pairs in turn, adding each
// view's geometric gradients (mean through the projection and the EWA
// Jacobian, scale and rotation or covariance, opacity, colour: 14 values)
// into the Gaussian's shared-memory sums with atomic adds.  The SH part is
// linear in each view's colour gradient: the Gaussian's own thread then runs
// it over its views with the 3M SH-gradient sums in registers, adds each
// view's direction term to the mean gradient and writes every output of its
// Gaussian (zeros when it is culled in every view).  The per-view
// screen-space gradient and the densification statistics (optional
// outputs) are handled by the same thread: all views' visibility bytes and
// 2D gradients are loaded at once (independent loads), then written out,
// zero where the Gaussian is not visible.
constexpr int ACC_SLOTS = 14;  // colour 3, opacity 1, mean 3, scale 3 + rotation 4 (or covariance 6)
constexpr int SP = BWD_BLOCK + 1;  // pitch of a slot's row of the block's Gaussians

// The Gaussian's sums: slot k of Gaussian t at acc[k * SP + t].
struct SlotSink {
  float *acc;  // + t
  __device__ __forceinline__ void mean2d(float, float) const {}
  __device__ __forceinline__ void color(int k, float v) const { atomicAdd(acc + k * SP, v); }
  __device__ __forceinline__ void opacity(float v) const { atomicAdd(acc + 3 * SP, v); }
  __device__ __forceinline__ void mean(int k, float v) const { atomicAdd(acc + (4 + k) * SP, v); }
  __device__ __forceinline__ void scale(int k, float v) const { atomicAdd(acc + (7 + k) * SP, v); }
  __device__ __forceinline__ void cov(int k, float v) const { atomicAdd(acc + (7 + k) * SP, v); }
  __device__ __forceinline__ void rot(float r, float x, float y, float z) const {
    atomicAdd(acc + 10 * SP, r); atomicAdd(acc + 11 * SP, x);
    atomicAdd(acc + 12 * SP, y); atomicAdd(acc + 13 * SP, z);
  }
};

// Bound by latency (SH rows, per-pair gathers).  VEC: the SH rows start on 16
// bytes (a multiple of four coefficients) and are read as float4.  16 views of
// 3M Gaussians: 951 us with a load per float and four blocks an SM; with float4
// 967 | 839 | 824 | 815 | 843 us at 4 | 5 | 6 | 7 | 8 blocks (spills from 6 on).
// Rows staged through shared memory both ways took 937 to 988 us: the staging
// takes the L1 that the pairs' gathers hit.
template <bool VEC>
__global__ void __launch_bounds__(BWD_BLOCK, 7)
preprocess_bwd_batched_kernel(const BatchViews bv, int P, int M, const float *__restrict__ means,
                              const float *__restrict__ shs, const float *__restrict__ scales,
                              const float *__restrict__ rots, const float *__restrict__ cov3D,
                              DmgsGrads out, int want_xy, float *__restrict__ densify_accum,
                              float *__restrict__ densify_count) {
  __shared__ float acc[ACC_SLOTS * SP];
  __shared__ uint32_t wsum[BWD_BLOCK / 32];
  __shared__ uint16_t pairs[BWD_BLOCK * MAX_BATCH_VIEWS];
  const int B = BWD_BLOCK;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int start = blockIdx.x * B;
  const int idx = start + t;
  for (int i = t; i < ACC_SLOTS * SP; i += B) acc[i] = 0.f;
  // per-view constants in shared memory: the pair loop below reads them
  // with a different view per lane, which from the kernel parameters would
  // be serialised constant-bank loads
  __shared__ ViewParams s_vp[MAX_BATCH_VIEWS];
  __shared__ float s_mat[MAX_BATCH_VIEWS][36];  // view matrix, projection matrix, camera centre
  __shared__ const float *s_gacc[MAX_BATCH_VIEWS];
  __shared__ const uint8_t *s_flags[MAX_BATCH_VIEWS];
  if (t < bv.nviews) {
    s_vp[t] = bv.v[t].vp;
    s_gacc[t] = bv.v[t].gacc;
    s_flags[t] = bv.v[t].flags;
  }
  for (int i = t; i < bv.nviews * 35; i += B) {
    const int v = i / 35, k = i - v * 35;
    const BatchView &W = bv.v[v];
    s_mat[v][k] = k < 16 ? __ldg(W.viewm + k) : (k < 32 ? __ldg(W.projm + k - 16) : __ldg(W.campos + k - 32));
  }
  uint32_t vm = 0u;
  uint8_t fl[MAX_BATCH_VIEWS];
  if (idx < P) {
#pragma unroll
    for (int v = 0; v < MAX_BATCH_VIEWS; ++v) fl[v] = v < bv.nviews ? bv.v[v].flags[idx] : 0u;
#pragma unroll
    for (int v = 0; v < MAX_BATCH_VIEWS; ++v) vm |= ((fl[v] & FLAG_VISIBLE) ? 1u : 0u) << v;
    if (want_xy) {
      float2 g2[MAX_BATCH_VIEWS];
#pragma unroll
      for (int v = 0; v < MAX_BATCH_VIEWS; ++v)
        g2[v] = ((vm >> v) & 1u) ? *reinterpret_cast<const float2 *>(bv.v[v].gacc + 12 * (size_t)idx)
                                 : make_float2(0.f, 0.f);
      float nsum = 0.f;
#pragma unroll
      for (int v = 0; v < MAX_BATCH_VIEWS; ++v) {
        if (v >= bv.nviews) break;
        float *d2 = bv.v[v].dL_dmeans2D;
        if (d2) {
          d2[3 * (size_t)idx] = g2[v].x;
          d2[3 * (size_t)idx + 1] = g2[v].y;
          d2[3 * (size_t)idx + 2] = 0.f;
        }
        if ((vm >> v) & 1u) nsum += sqrtf(g2[v].x * g2[v].x + g2[v].y * g2[v].y);
      }
      if (densify_accum && vm) {
        densify_accum[idx] += nsum;
        densify_count[idx] += (float)__popc(vm);
      }
    }
  }
  // block-wide exclusive scan of the pair counts
  const uint32_t cnt = __popc(vm);
  uint32_t inc = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) wsum[wid] = inc;
  __syncthreads();
  uint32_t off = inc - cnt, total = 0;
#pragma unroll
  for (int w = 0; w < BWD_BLOCK / 32; ++w) {
    off += w < wid ? wsum[w] : 0u;
    total += wsum[w];
  }
  for (uint32_t m = vm; m; m &= m - 1) pairs[off++] = (uint16_t)((t << 4) | (__ffs(m) - 1));
  __syncthreads();
  for (uint32_t i = t; i < total; i += B) {
    const uint32_t pr = pairs[i];
    const int gl = (int)(pr >> 4), v = (int)(pr & 15u);
    const ViewParams vp = s_vp[v];
    const SlotSink sink{acc + gl};
    float pm[3], prgb[3];
    preprocess_bwd_one(start + gl, vp, s_mat[v], s_mat[v] + 16, means, scales, rots, cov3D, s_gacc[v],
                       out, sink, pm, prgb);
    if (out.dL_dmeans3D)
#pragma unroll
      for (int k = 0; k < 3; ++k) sink.mean(k, pm[k]);
  }
  __syncthreads();
  if (idx >= P) return;

  // --- the Gaussian's own thread: SH over its views, then every output ---
  const float *own = acc + t;
  float dm[3] = {own[4 * SP], own[5 * SP], own[6 * SP]};
  const bool want_sh = shs != nullptr && (out.dL_dsh != nullptr || out.dL_dmeans3D != nullptr);
  float dsh[48];
#pragma unroll
  for (int i = 0; i < 48; ++i) dsh[i] = 0.f;
  if (want_sh && vm) {
    const float mx = means[3 * (size_t)idx], my = means[3 * (size_t)idx + 1],
                mz = means[3 * (size_t)idx + 2];
    const float *sh = shs + (size_t)idx * M * 3;
    for (uint32_t m = vm; m; m &= m - 1) {
      const int v = __ffs(m) - 1;
      const float *gv = s_gacc[v] + 12 * (size_t)idx;
      float drgb[3] = {gv[6], gv[7], gv[8]};
      apply_clamp(s_flags[v][idx], drgb);
      // four coefficients' twelve floats as three float4 where rows start on
      // 16 bytes: lanes read different rows, a wavefront a lane and load
      float4 q0, q1, q2;
      sh_bwd(s_vp[v].D, mx, my, mz, s_mat[v] + 32, drgb,
             [&](int j) {
               if (!VEC) return sh[j];
               if (j % 12 == 0) {
                 q0 = __ldg(reinterpret_cast<const float4 *>(sh + j));
                 q1 = __ldg(reinterpret_cast<const float4 *>(sh + j) + 1);
                 q2 = __ldg(reinterpret_cast<const float4 *>(sh + j) + 2);
               }
               const float4 q = j % 12 < 4 ? q0 : j % 12 < 8 ? q1 : q2;
               return j % 4 == 0 ? q.x : j % 4 == 1 ? q.y : j % 4 == 2 ? q.z : q.w;
             },
             [&](int j, float x) { dsh[j] += x; }, dm);
    }
  }
  const size_t i3 = 3 * (size_t)idx;
  if (out.dL_dcolors) {
    out.dL_dcolors[i3] = own[0]; out.dL_dcolors[i3 + 1] = own[SP]; out.dL_dcolors[i3 + 2] = own[2 * SP];
  }
  if (out.dL_dopacity) out.dL_dopacity[idx] = own[3 * SP];
  if (out.dL_dmeans3D) {
    out.dL_dmeans3D[i3] = dm[0]; out.dL_dmeans3D[i3 + 1] = dm[1]; out.dL_dmeans3D[i3 + 2] = dm[2];
  }
  if (out.dL_dcov3D) {
#pragma unroll
    for (int k = 0; k < 6; ++k) out.dL_dcov3D[6 * (size_t)idx + k] = own[(7 + k) * SP];
  }
  if (out.dL_dscales) {
    out.dL_dscales[i3] = own[7 * SP]; out.dL_dscales[i3 + 1] = own[8 * SP]; out.dL_dscales[i3 + 2] = own[9 * SP];
  }
  if (out.dL_drotations)
    reinterpret_cast<float4 *>(out.dL_drotations)[idx] =
        make_float4(own[10 * SP], own[11 * SP], own[12 * SP], own[13 * SP]);
  if (out.dL_dsh) {
    // the Gaussian's 3M contiguous floats: coefficients above degree 3 (or
    // the active degree) stay zero
    float *d = out.dL_dsh + (size_t)idx * M * 3;
    const int n = 3 * M;
    if (n >= 48 && (n & 3) == 0 && (reinterpret_cast<uintptr_t>(d) & 15) == 0) {
      float4 *d4 = reinterpret_cast<float4 *>(d);
#pragma unroll
      for (int i = 0; i < 12; ++i) d4[i] = make_float4(dsh[4 * i], dsh[4 * i + 1], dsh[4 * i + 2], dsh[4 * i + 3]);
      for (int i = 12; i < (n >> 2); ++i) d4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
#pragma unroll
      for (int i = 0; i < 48; ++i)
        if (i < n) d[i] = dsh[i];
      for (int i = 48; i < n; ++i) d[i] = 0.f;
    }
  }
}

}  // namespace

ZeroSpans preprocess_bwd_outputs(const DmgsGrads &out, int P, int M) {
  ZeroSpans z;
  const size_t n = P > 0 ? (size_t)P : 0;
  z.add(out.dL_dmeans2D, 3 * n);
  z.add(out.dL_dcolors, 3 * n);
  z.add(out.dL_dopacity, n);
  z.add(out.dL_dmeans3D, 3 * n);
  z.add(out.dL_dcov3D, 6 * n);
  z.add(out.dL_dscales, 3 * n);
  z.add(out.dL_drotations, 4 * n);
  z.add(out.dL_dsh, 3 * (size_t)std::max(M, 0) * n);
  return z;
}

int launch_preprocess_bwd(const ViewParams &vp, const float *viewm, const float *projm,
                          const float *campos, const GaussianPtrs &g, const GeomLayout &L,
                          const char *geom, const float *gacc, const DmgsGrads &out,
                          cudaStream_t s) {
  if (g.P <= 0) return DMGS_OK;
  const size_t smem = (size_t)BWD_BLOCK * SHP * 4;
  // the visible count is known on the device alone: a few waves of blocks
  // stride over the list
  const int grid = std::min((g.P + BWD_BLOCK - 1) / BWD_BLOCK, 16 * NUM_SMS_HINT);
  DMGS_TIMED(K_PREPROCESS_BWD, s, dmgs_host::note_launch(), preprocess_bwd_list_kernel<<<grid, BWD_BLOCK, smem, s>>>(
      vp, viewm, projm, campos, g.P, g.M, g.means3D, g.shs, g.scales, g.rotations, g.cov3D,
      reinterpret_cast<const uint8_t *>(geom + L.flags), gacc,
      reinterpret_cast<const uint32_t *>(geom + L.vlist),
      reinterpret_cast<const uint32_t *>(geom + L.counters), out));
  DMGS_LAUNCH_CHECK("preprocess_bwd_list_kernel");
  return DMGS_OK;
}

}  // namespace dmgs

namespace dmgs {

int launch_preprocess_bwd_batched(const BatchViews &bv, const GaussianPtrs &g, const DmgsGrads &out,
                                  float *densify_accum, float *densify_count, cudaStream_t s) {
  if (g.P <= 0) return DMGS_OK;
  int want_xy = densify_accum != nullptr;
  for (int v = 0; v < bv.nviews; ++v) want_xy |= bv.v[v].dL_dmeans2D != nullptr;
  const bool vec = (g.M & 3) == 0 && (reinterpret_cast<uintptr_t>(g.shs) & 15) == 0;
  const auto kernel = vec ? preprocess_bwd_batched_kernel<true> : preprocess_bwd_batched_kernel<false>;
  DMGS_TIMED(K_BATCH_PREPROCESS_BWD, s, dmgs_host::note_launch(),
             kernel<<<(g.P + BWD_BLOCK - 1) / BWD_BLOCK, BWD_BLOCK, 0, s>>>(
                 bv, g.P, g.M, g.means3D, g.shs, g.scales, g.rotations, g.cov3D, out, want_xy, densify_accum,
                 densify_count));
  DMGS_LAUNCH_CHECK("preprocess_bwd_batched_kernel");
  return DMGS_OK;
}

}  // namespace dmgs
