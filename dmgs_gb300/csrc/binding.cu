// binding.cu — mesh -> Gaussian face binding and its adjoint.
//
// Stage-2 form: scene/gaussian_geo_model_mlp_flex.py:258-335 (renew_gaussian)
// and :370-385 (get_covariance_dyn), with the frame of geo/mesh_utils.py:43-57.
// The reference evaluates it as ~40 separate torch ops per step.
//
// The kernels are bound by memory, and a thread per face looping over its
// Gaussians' rows in global memory touched each array G rows apart per lane:
// every 32-byte sector moved several times (700k faces, G = 6, stage 3: 206
// us forward and 195 us adjoint, against 82 and 150; floors 39 and 35).
// Rows now pass through shared memory, a warp's accesses consecutive.
// A thread per face walks its Gaussians in order, 64 faces a block, on the
// block's staged rows.  Where fewer faces fit, the stage-3 kernels, whose
// arithmetic is per Gaussian, share a face's Gaussians among the threads left
// over (2M Gaussians, both directions, at 24 | 64 | 128 | 512 per face: 404 |
// 405 | 807 | 3307 us with a thread per face on global rows, 273 | 581 | 1019 |
// 2632 us with one on staged rows, 125 | 141 | 139 | 199 us so).  (A thread
// per Gaussian, with the faces formed by the block's first 128 / G threads:
// three warps in four waited at the barriers, 90 and 240 us.)
//
// Stage-3 form: scene/gaussian_geo_model_finetune.py:396-421 (renew_gaussian)
// and :446-483 (get_scaling / get_rotation / get_rot_matrix).  The rotation
// matrix -> quaternion step uses Shepperd's method (pick the largest of
// trace, R00, R11, R22 to divide by), made sign-unique by a non-negative real
// part, then normalised — the same function the reference obtains from
// pytorch3d's matrix_to_quaternion followed by F.normalize.
#include <algorithm>

#include "kernels.cuh"

namespace dmgs {

namespace {

struct f3 { float x, y, z; };
__device__ __forceinline__ f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 operator*(float s, f3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 cross(f3 a, f3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ f3 shfl_xor(f3 a, int o) {
  return {__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o), __shfl_xor_sync(0xffffffffu, a.z, o)};
}
__device__ __forceinline__ float norm(f3 a) { return sqrtf(dot(a, a)); }

constexpr float NRM_EPS = 1e-12f;  // torch.nn.functional.normalize default eps

// Faces whose vertex indices leave [0, V) are skipped (their outputs are
// left as written by the caller; no gradient is scattered).
__device__ __forceinline__ bool face_ok(int64_t i0, int64_t i1, int64_t i2, int V) {
  return i0 >= 0 && i1 >= 0 && i2 >= 0 && i0 < V && i1 < V && i2 < V;
}

__device__ __forceinline__ f3 load_v(const float *verts, int64_t i) {
  return mk(verts[3 * i], verts[3 * i + 1], verts[3 * i + 2]);
}

// unit(v) = v / max(|v|, eps) and its adjoint.
__device__ __forceinline__ f3 unit(f3 v, float &len) {
  len = norm(v);
  return (1.f / fmaxf(len, NRM_EPS)) * v;
}
__device__ __forceinline__ f3 unit_adj(f3 u, float len, f3 g) {
  if (len > NRM_EPS) return (1.f / len) * (g - dot(u, g) * u);
  return (1.f / NRM_EPS) * g;
}

struct Frame {
  f3 e01, e02, x, y, n, nraw, u;
  float len, nlen, ulen;
};

__device__ __forceinline__ Frame face_frame(f3 v0, f3 v1, f3 v2) {
  Frame F;
  F.e01 = v1 - v0;
  F.e02 = v2 - v0;
  F.x = unit(F.e01, F.len);
  F.nraw = cross(F.e01, F.e02);
  F.n = unit(F.nraw, F.nlen);
  F.u = cross(F.n, F.x);
  F.y = unit(F.u, F.ulen);
  return F;
}

// Adjoint of the frame: gradients w.r.t. x, y, n -> w.r.t. v0, v1, v2.
__device__ __forceinline__ void face_frame_adj(const Frame &F, f3 gx, f3 gy, f3 gn, f3 &g0,
                                               f3 &g1, f3 &g2) {
  const f3 gu = unit_adj(F.y, F.ulen, gy);
  gn = gn + cross(F.x, gu);       // u = n x x
  gx = gx + cross(gu, F.n);
  const f3 gnr = unit_adj(F.n, F.nlen, gn);
  f3 ge01 = cross(F.e02, gnr);    // nraw = e01 x e02
  f3 ge02 = cross(gnr, F.e01);
  ge01 = ge01 + unit_adj(F.x, F.len, gx);
  g1 = ge01;
  g2 = ge02;
  g0 = mk(0.f, 0.f, 0.f) - ge01 - ge02;
}

// Triangle-space factor L (3x3 row-major) of the stage-2 covariance.
__device__ __forceinline__ void tri_L(const Frame &F, float rad_base, float z_scale, int adaptive,
                                      float *L) {
  const float len = fmaxf(F.len, NRM_EPS);
  float m01 = 0.f, m11 = 1.f;
  if (adaptive) {
    const float Ax = dot(F.e02, F.x), Ay = dot(F.e02, F.y);
    const float Ex = len * 0.5f, Ey = len * 0.8660254037844386f;  // sqrt(3)/2
    m01 = (Ax - Ex) / Ey;
    m11 = Ay / Ey;
  }
  const float s = len * rad_base;
  L[0] = s;   L[1] = m01 * s; L[2] = 0.f;
  L[3] = 0.f; L[4] = m11 * s; L[5] = 0.f;
  L[6] = 0.f; L[7] = 0.f;     L[8] = z_scale;
}

__device__ __forceinline__ float bc_at(const DmgsFaceBinding &b, int f, int g, int k) {
  return b.bc_per_gaussian ? b.bc[((size_t)f * b.G + g) * 3 + k] : b.bc[g * 3 + k];
}

// ---- the blocks of the four kernels ---------------------------------------------

constexpr int BB = 64;  // threads, and faces per block

// Rows of a block: the faces it takes and the Gaussians of each that
// its shared memory holds at a time (all of them, or, with one face, a part),
// and the threads that share a face's Gaussians (stage 3: a power of two, lanes
// of one warp).
struct FaceBlocks {
  int faces, chunk, blocks, share;
  size_t smem;
};

FaceBlocks face_blocks(int F, int G, int words) {
  FaceBlocks k;
  // Gaussians whose rows fit (64 faces of six: ten blocks share an SM)
  const int fit = 22 * 1024 / 4 / words;
  k.faces = std::max(1, std::min(BB, fit / G));
  k.chunk = std::min(G, fit);
  k.blocks = (F + k.faces - 1) / k.faces;
  k.share = 1;
  while (2 * k.share * k.faces <= BB && k.share < 32) k.share *= 2;
  k.smem = (size_t)k.faces * k.chunk * words * 4 + 5 * 16;  // each array padded to 16 bytes
  return k;
}

// The next of the consecutive arrays in a block's shared memory.
__device__ __forceinline__ float *take(float *&p, int floats) {
  float *q = p;
  p += (floats + 3) & ~3;
  return q;
}

// n floats of consecutive rows between global and shared memory.
__device__ __forceinline__ void rows_in(const float *__restrict__ g, int n, float *sm) {
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
    for (int i = threadIdx.x; i < n / 4; i += BB)
      reinterpret_cast<float4 *>(sm)[i] = __ldg(reinterpret_cast<const float4 *>(g) + i);
    for (int i = (n & ~3) + threadIdx.x; i < n; i += BB) sm[i] = __ldg(g + i);
  } else {
    for (int i = threadIdx.x; i < n; i += BB) sm[i] = __ldg(g + i);
  }
}
__device__ __forceinline__ void rows_out(float *__restrict__ g, int n, const float *sm) {
  if ((reinterpret_cast<uintptr_t>(g) & 15) == 0) {
    for (int i = threadIdx.x; i < n / 4; i += BB)
      reinterpret_cast<float4 *>(g)[i] = reinterpret_cast<const float4 *>(sm)[i];
    for (int i = (n & ~3) + threadIdx.x; i < n; i += BB) g[i] = sm[i];
  } else {
    for (int i = threadIdx.x; i < n; i += BB) g[i] = sm[i];
  }
}
// A face's triangle; false when an index is out of range.
struct Tri {
  int64_t i0, i1, i2;
  f3 v0, v1, v2;
};
__device__ __forceinline__ bool load_tri(const int64_t *__restrict__ faces, const float *__restrict__ verts, int V, int f,
                                         Tri &T) {
  T.i0 = faces[3 * (size_t)f]; T.i1 = faces[3 * (size_t)f + 1]; T.i2 = faces[3 * (size_t)f + 2];
  if (!face_ok(T.i0, T.i1, T.i2, V)) return false;
  T.v0 = load_v(verts, T.i0); T.v1 = load_v(verts, T.i1); T.v2 = load_v(verts, T.i2);
  return true;
}

__device__ __forceinline__ void scatter_vertices(float *__restrict__ dverts, const Tri &T, f3 g0, f3 g1, f3 g2) {
  atomicAdd(dverts + 3 * T.i0, g0.x); atomicAdd(dverts + 3 * T.i0 + 1, g0.y); atomicAdd(dverts + 3 * T.i0 + 2, g0.z);
  atomicAdd(dverts + 3 * T.i1, g1.x); atomicAdd(dverts + 3 * T.i1 + 1, g1.y); atomicAdd(dverts + 3 * T.i1 + 2, g1.z);
  atomicAdd(dverts + 3 * T.i2, g2.x); atomicAdd(dverts + 3 * T.i2 + 1, g2.y); atomicAdd(dverts + 3 * T.i2 + 2, g2.z);
}

// ----------------------------- stage 2 -----------------------------------

__global__ void __launch_bounds__(BB)
bind_fwd_kernel(DmgsFaceBinding b, FaceBlocks kb, float *__restrict__ xyz, float *__restrict__ cov,
                float *__restrict__ rot, float *__restrict__ covL) {
  extern __shared__ __align__(16) float bind_smem[];
  const int t = threadIdx.x, f0 = blockIdx.x * kb.faces, nf = min(kb.faces, b.F - f0), f = f0 + t;
  float *p = bind_smem;
  float *sx = take(p, 3 * kb.faces * kb.chunk), *sc = take(p, 6 * kb.faces * kb.chunk);
  Tri T;
  float c[6];
  bool good = true;
  if (t < nf) {
    good = load_tri(b.faces, b.verts, b.V, f, T);
    if (good) {
      const Frame F = face_frame(T.v0, T.v1, T.v2);
      float L[9];
      tri_L(F, b.rad_base, b.z_scale, b.adaptive_cov, L);
      // no scale factor: the real-scene variant's covariance, L unscaled
      // (scene/gaussian_geo_model_mlp_flex_colmap.py:494-512)
      const float k = b.scale_factor ? tanhf(b.scale_factor[0]) * b.max_scale : 1.f;
      const float R[9] = {F.x.x, F.y.x, F.n.x, F.x.y, F.y.y, F.n.y, F.x.z, F.y.z, F.n.z};
      float Mf[9];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          Mf[i * 3 + j] = k * (R[i * 3] * L[j] + R[i * 3 + 1] * L[3 + j] + R[i * 3 + 2] * L[6 + j]);
      auto sig = [&](int i, int j) {
        return Mf[i * 3] * Mf[j * 3] + Mf[i * 3 + 1] * Mf[j * 3 + 1] + Mf[i * 3 + 2] * Mf[j * 3 + 2];
      };
      c[0] = sig(0, 0); c[1] = sig(0, 1); c[2] = sig(0, 2); c[3] = sig(1, 1); c[4] = sig(1, 2); c[5] = sig(2, 2);
      if (rot)
        for (int i = 0; i < 9; ++i) rot[(size_t)f * 9 + i] = R[i];
      if (covL)
        for (int i = 0; i < 9; ++i) covL[(size_t)f * 9 + i] = L[i];
    }
  }
  const bool all_good = __syncthreads_and(good);
  for (int gs = 0; gs < b.G; gs += kb.chunk) {  // once, unless one face's rows do not fit
    const int gn = min(kb.chunk, b.G - gs), m = nf * gn;
    const size_t o0 = (size_t)f0 * b.G + gs;
    if (good && t < nf) {
      for (int g = 0; g < gn; ++g) {
        const int q = t * gn + g;
        const float w0 = bc_at(b, f, gs + g, 0), w1 = bc_at(b, f, gs + g, 1), w2 = bc_at(b, f, gs + g, 2);
        const float x = w0 * T.v0.x + w1 * T.v1.x + w2 * T.v2.x, y = w0 * T.v0.y + w1 * T.v1.y + w2 * T.v2.y;
        const float z = w0 * T.v0.z + w1 * T.v1.z + w2 * T.v2.z;
        if (all_good) {
          sx[3 * q] = x; sx[3 * q + 1] = y; sx[3 * q + 2] = z;
#pragma unroll
          for (int i = 0; i < 3; ++i) reinterpret_cast<float2 *>(sc)[3 * q + i] = make_float2(c[2 * i], c[2 * i + 1]);
        } else {  // a skipped face's outputs stay as the caller left them
          const size_t o = o0 + q;
          if (xyz) { xyz[3 * o] = x; xyz[3 * o + 1] = y; xyz[3 * o + 2] = z; }
          if (cov)
#pragma unroll
            for (int i = 0; i < 6; ++i) cov[6 * o + i] = c[i];
        }
      }
    }
    __syncthreads();
    if (all_good) {
      if (xyz) rows_out(xyz + 3 * o0, 3 * m, sx);
      if (cov) rows_out(cov + 6 * o0, 6 * m, sc);
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(BB)
bind_bwd_kernel(DmgsFaceBinding b, FaceBlocks kb, const float *__restrict__ dxyz,
                const float *__restrict__ dcov, float *__restrict__ dverts,
                float *__restrict__ dsf) {
  extern __shared__ __align__(16) float bind_smem[];
  const int t = threadIdx.x, f0 = blockIdx.x * kb.faces, nf = min(kb.faces, b.F - f0), f = f0 + t;
  float *p = bind_smem;
  float *sx = take(p, 3 * kb.faces * kb.chunk), *sc = take(p, 6 * kb.faces * kb.chunk);
  Tri T;
  bool good = false;
  f3 g0 = mk(0.f, 0.f, 0.f), g1 = g0, g2 = g0;
  float gc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int gs = 0; gs < b.G; gs += kb.chunk) {  // once, unless one face's rows do not fit
    const int gn = min(kb.chunk, b.G - gs), m = nf * gn;
    const size_t o = (size_t)f0 * b.G + gs;
    if (dxyz) rows_in(dxyz + 3 * o, 3 * m, sx);
    if (dcov) rows_in(dcov + 6 * o, 6 * m, sc);
    if (gs == 0 && t < nf) good = load_tri(b.faces, b.verts, b.V, f, T);
    __syncthreads();
    if (good) {
      for (int g = 0; g < gn; ++g) {
        const int q = t * gn + g;
        if (dxyz) {
          const f3 d = mk(sx[3 * q], sx[3 * q + 1], sx[3 * q + 2]);
          g0 = g0 + bc_at(b, f, gs + g, 0) * d;
          g1 = g1 + bc_at(b, f, gs + g, 1) * d;
          g2 = g2 + bc_at(b, f, gs + g, 2) * d;
        }
        if (dcov)
#pragma unroll
          for (int i = 0; i < 6; ++i) gc[i] += sc[6 * q + i];
      }
    }
    __syncthreads();
  }
  float dk_local = 0.f;
  if (good) {
    if (dcov) {
      const Frame F = face_frame(T.v0, T.v1, T.v2);
      float L[9];
      tri_L(F, b.rad_base, b.z_scale, b.adaptive_cov, L);
      const float th = b.scale_factor ? tanhf(b.scale_factor[0]) : 0.f;
      const float k = b.scale_factor ? th * b.max_scale : 1.f;
      const float R[9] = {F.x.x, F.y.x, F.n.x, F.x.y, F.y.y, F.n.y, F.x.z, F.y.z, F.n.z};
      float RL[9];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          RL[i * 3 + j] = R[i * 3] * L[j] + R[i * 3 + 1] * L[3 + j] + R[i * 3 + 2] * L[6 + j];
      // symmetric gradient of the packed covariance
      const float Gs[9] = {gc[0], 0.5f * gc[1], 0.5f * gc[2], 0.5f * gc[1], gc[3],
                           0.5f * gc[4], 0.5f * gc[2], 0.5f * gc[4], gc[5]};
      // dMf = 2 Gs Mf, Mf = k RL
      float dMf[9];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          dMf[i * 3 + j] = 2.f * k * (Gs[i * 3] * RL[j] + Gs[i * 3 + 1] * RL[3 + j] + Gs[i * 3 + 2] * RL[6 + j]);
      float dk = 0.f;
#pragma unroll
      for (int i = 0; i < 9; ++i) dk += dMf[i] * RL[i];
      if (b.scale_factor) dk_local = dk * b.max_scale * (1.f - th * th);
      // dR = dMf (k L)^T
      float dR[9];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          dR[i * 3 + j] = k * (dMf[i * 3] * L[j * 3] + dMf[i * 3 + 1] * L[j * 3 + 1] + dMf[i * 3 + 2] * L[j * 3 + 2]);
      const f3 gxv = mk(dR[0], dR[3], dR[6]);
      const f3 gyv = mk(dR[1], dR[4], dR[7]);
      const f3 gnv = mk(dR[2], dR[5], dR[8]);
      f3 h0, h1, h2;
      face_frame_adj(F, gxv, gyv, gnv, h0, h1, h2);
      g0 = g0 + h0; g1 = g1 + h1; g2 = g2 + h2;
    }
    scatter_vertices(dverts, T, g0, g1, g2);
  }
  if (dsf) {
    const float s = warp_sum(dk_local);
    if ((threadIdx.x & 31) == 0 && s != 0.f) atomicAdd(dsf, s);
  }
}

// ----------------------------- stage 3 -----------------------------------

// 1 / sqrt(x) for positive normal x: the hardware's estimate and one
// Newton-Raphson step (within an ulp; a root and a division each cost some
// thirty instructions with their special cases, and a Gaussian needs three).
__device__ __forceinline__ float inv_sqrt(float x) {
  const float y = rsqrtf(x);
  return fmaf(fmaf(-x * y, y, 1.f), 0.5f * y, y);
}

// 1 / max(sqrt(x), NRM_EPS) for finite x >= 0 (the guard of torch's normalize).
__device__ __forceinline__ float inv_norm(float x) {
  return x > NRM_EPS * NRM_EPS ? inv_sqrt(x) : 1.f / NRM_EPS;
}

// The same of a caller's pair, whose squares may overflow: 0 then (the
// Newton-Raphson step would give inf * 0).
__device__ __forceinline__ float inv_norm2(float a, float b) {
  const float x = a * a + b * b, r = inv_norm(x);
  return x < __int_as_float(0x7f800000) || x != x ? r : 0.f;
}

// Unit quaternion (w, x, y, z), w >= 0, of a rotation matrix (row-major),
// Shepperd's method: with big the largest component, half the root of its
// arg, the others are K[big][c] 0.25 / max(big, 0.05), where K[0][c] are the
// differences and the rest the sums of mirrored entries.  Every choice is a
// select (a warp's lanes differ in it); the reciprocals are kept for the
// adjoint.
struct QuatOut { float q[4]; int br; float sgn, big, d, inv; };

// Component c of the K row of the largest component br (0 for c == br).
__device__ __forceinline__ float quat_k(const float *R, int br, int c) {
  const float k01 = R[7] - R[5], k02 = R[2] - R[6], k03 = R[3] - R[1];
  const float k12 = R[1] + R[3], k13 = R[2] + R[6], k23 = R[5] + R[7];
  if (c == 0) return br == 1 ? k01 : (br == 2 ? k02 : (br == 3 ? k03 : 0.f));
  if (c == 1) return br == 0 ? k01 : (br == 2 ? k12 : (br == 3 ? k13 : 0.f));
  if (c == 2) return br == 0 ? k02 : (br == 1 ? k12 : (br == 3 ? k23 : 0.f));
  return br == 0 ? k03 : (br == 1 ? k13 : (br == 2 ? k23 : 0.f));
}

__device__ __forceinline__ QuatOut mat_to_quat(const float *R) {
  QuatOut o;
  const float tr = R[0] + R[4] + R[8];
  o.br = (tr >= R[0] && tr >= R[4] && tr >= R[8]) ? 0 : (R[0] >= R[4] && R[0] >= R[8]) ? 1 : (R[4] >= R[8]) ? 2 : 3;
  const float s0 = o.br < 2 ? R[0] : -R[0], s4 = (o.br & 1) ? -R[4] : R[4], s8 = (o.br == 0 || o.br == 3) ? R[8] : -R[8];
  const float arg = fmaxf(o.br == 0 ? 1.f + tr : 1.f + s0 + s4 + s8, 0.f);
  const float ia = inv_sqrt(fmaxf(arg, 1e-30f));
  o.big = 0.5f * (arg * ia);
  o.d = o.big < 0.05f ? 0.25f / 0.05f : 0.5f * ia;  // 0.25 / max(big, 0.05)
  float raw[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) raw[c] = c == o.br ? o.big : quat_k(R, o.br, c) * o.d;
  o.sgn = raw[0] < 0.f ? -1.f : 1.f;
  o.inv = inv_norm(raw[0] * raw[0] + raw[1] * raw[1] + raw[2] * raw[2] + raw[3] * raw[3]);
#pragma unroll
  for (int c = 0; c < 4; ++c) o.q[c] = o.sgn * raw[c] * o.inv;
  return o;
}

// Adjoint of mat_to_quat: dq (w.r.t. the normalised output) -> dR.
__device__ __forceinline__ void mat_to_quat_adj(const float *R, const QuatOut &o, const float *dq,
                                                float *dR) {
  float dr[4];
  const float qd = o.q[0] * dq[0] + o.q[1] * dq[1] + o.q[2] * dq[2] + o.q[3] * dq[3];
#pragma unroll
  for (int c = 0; c < 4; ++c)  // w.r.t. the pre-sign (w, x, y, z)
    dr[c] = o.sgn * ((o.inv < 1.f / NRM_EPS ? dq[c] - o.q[c] * qd : dq[c]) * o.inv);
  float dd = 0.f, dk[4], dbig = 0.f;  // gradients w.r.t. d and the K row
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const bool own = c == o.br;
    dd += own ? 0.f : dr[c] * quat_k(R, o.br, c);
    dk[c] = own ? 0.f : dr[c] * o.d;
    dbig = own ? dr[c] : dbig;
  }
  // d = 0.25 / big -> -0.25 / big^2 = -4 d^2; big = 0.5 sqrt(arg) -> 0.125 / big
  float darg;
  if (!(o.big < 0.05f)) {
    dbig += dd * (-4.f * o.d * o.d);
    darg = dbig * (0.5f * o.d);
  } else {  // d is clamped
    darg = o.big > 0.f ? dbig * 0.125f / o.big : 0.f;
  }
  const float e01 = o.br == 0 ? dk[1] : (o.br == 1 ? dk[0] : 0.f), e02 = o.br == 0 ? dk[2] : (o.br == 2 ? dk[0] : 0.f);
  const float e03 = o.br == 0 ? dk[3] : (o.br == 3 ? dk[0] : 0.f), e12 = o.br == 1 ? dk[2] : (o.br == 2 ? dk[1] : 0.f);
  const float e13 = o.br == 1 ? dk[3] : (o.br == 3 ? dk[1] : 0.f), e23 = o.br == 2 ? dk[3] : (o.br == 3 ? dk[2] : 0.f);
  dR[0] = o.br < 2 ? darg : -darg;
  dR[4] = (o.br & 1) ? -darg : darg;
  dR[8] = (o.br == 0 || o.br == 3) ? darg : -darg;
  dR[7] = e01 + e23; dR[5] = e23 - e01;
  dR[2] = e02 + e13; dR[6] = e13 - e02;
  dR[3] = e03 + e12; dR[1] = e12 - e03;
}

// STAGED: the rows through shared memory, as above.  With up to three Gaussians
// per face a thread's rows in global memory are short enough for neighbouring
// lanes to share their sectors, and more blocks an SM count for more: 2M
// Gaussians, both directions, staged | direct, 264 | 156 us at one per face,
// 178 | 119 at two, 143 | 133 at three, 138 | 152 at four; 60,000: 20.5 | 18.5,
// 21.3 | 18.5, 24.6 | 22.6, 23.6 | 23.6.  Blocks an SM of the direct form, at
// one per face: 189 | 174 | 154 | 162 us at 10 | 12 | 16 | 20.
constexpr int DIRECT_MAX = 3;

template <bool STAGED>
__global__ void __launch_bounds__(BB, STAGED ? 10 : 16)
bind3_fwd_kernel(DmgsFaceBinding3 b, FaceBlocks kb, float *__restrict__ xyz,
                 float *__restrict__ scales, float *__restrict__ rots) {
  extern __shared__ __align__(16) float bind_smem[];
  // thread t: face t / share of the block, its Gaussians sub, sub + share, ...
  const int t = threadIdx.x / kb.share, sub = threadIdx.x % kb.share;
  const int f0 = blockIdx.x * kb.faces, nf = min(kb.faces, b.F - f0), cap = kb.faces * kb.chunk;
  float *p = bind_smem;
  float *sq = take(p, 4 * cap), *sx = take(p, 3 * cap), *ss = take(p, 3 * cap), *s2 = take(p, 2 * cap), *r2 = take(p, 2 * cap);
  Tri T;
  float Rw[9];
  bool good = true;
  for (int gs = 0; gs < b.G; gs += kb.chunk) {  // once, unless one face's rows do not fit
    const int gn = min(kb.chunk, b.G - gs), m = nf * gn;
    const size_t o0 = (size_t)f0 * b.G + gs;
    const float *in_s2 = STAGED ? s2 : b.scaling2d + 2 * o0, *in_r2 = STAGED ? r2 : b.rotation2d + 2 * o0;
    if (STAGED) {
      if (scales) rows_in(b.scaling2d + 2 * o0, 2 * m, s2);
      if (rots) rows_in(b.rotation2d + 2 * o0, 2 * m, r2);
    }
    if (gs == 0 && t < nf) {
      good = load_tri(b.faces, b.verts, b.V, f0 + t, T);
      if (good) {
        const Frame F = face_frame(T.v0, T.v1, T.v2);
        const float R[9] = {F.x.x, F.y.x, F.n.x, F.x.y, F.y.y, F.n.y, F.x.z, F.y.z, F.n.z};
#pragma unroll
        for (int i = 0; i < 9; ++i) Rw[i] = R[i];
      }
    }
    const bool all_good = STAGED && __syncthreads_and(good);
    if (good && t < nf) {
      for (int g = sub; g < gn; g += kb.share) {
        const int q = t * gn + g;
        const float *w = b.bc + 3 * (gs + g);
        const float w0 = w[0], w1 = w[1], w2 = w[2];
        const float x = w0 * T.v0.x + w1 * T.v1.x + w2 * T.v2.x, y = w0 * T.v0.y + w1 * T.v1.y + w2 * T.v2.y;
        const float z = w0 * T.v0.z + w1 * T.v1.z + w2 * T.v2.z;
        float e0 = 0.f, e1 = 0.f;
        if (scales) {
          e0 = expf(in_s2[2 * q]);
          e1 = expf(in_s2[2 * q + 1]);
        }
        float4 quat = make_float4(0.f, 0.f, 0.f, 0.f);
        if (rots) {
          const float ra = in_r2[2 * q], rb = in_r2[2 * q + 1];
          const float cn = inv_norm2(ra, rb);
          const float a = ra * cn, s = rb * cn;
          // R = Rw * [[a,-s,0],[s,a,0],[0,0,1]]
          float R[9];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            R[i * 3 + 0] = Rw[i * 3] * a + Rw[i * 3 + 1] * s;
            R[i * 3 + 1] = -Rw[i * 3] * s + Rw[i * 3 + 1] * a;
            R[i * 3 + 2] = Rw[i * 3 + 2];
          }
          const QuatOut o = mat_to_quat(R);
          quat = make_float4(o.q[0], o.q[1], o.q[2], o.q[3]);
        }
        if (all_good) {
          sx[3 * q] = x; sx[3 * q + 1] = y; sx[3 * q + 2] = z;
          ss[3 * q] = e0; ss[3 * q + 1] = e1; ss[3 * q + 2] = b.thin_z;
          reinterpret_cast<float4 *>(sq)[q] = quat;
        } else {  // a skipped face's outputs stay as the caller left them
          const size_t o = o0 + q;
          if (xyz) { xyz[3 * o] = x; xyz[3 * o + 1] = y; xyz[3 * o + 2] = z; }
          if (scales) { scales[3 * o] = e0; scales[3 * o + 1] = e1; scales[3 * o + 2] = b.thin_z; }
          if (rots) { rots[4 * o] = quat.x; rots[4 * o + 1] = quat.y; rots[4 * o + 2] = quat.z; rots[4 * o + 3] = quat.w; }
        }
      }
    }
    if (STAGED) __syncthreads();
    if (all_good) {
      if (xyz) rows_out(xyz + 3 * o0, 3 * m, sx);
      if (scales) rows_out(scales + 3 * o0, 3 * m, ss);
      if (rots) rows_out(rots + 4 * o0, 4 * m, sq);
      __syncthreads();
    }
  }
}

template <bool STAGED>
__global__ void __launch_bounds__(BB, STAGED ? 10 : 16)
bind3_bwd_kernel(DmgsFaceBinding3 b, FaceBlocks kb, const float *__restrict__ dxyz,
                 const float *__restrict__ dscales, const float *__restrict__ drots,
                 float *__restrict__ dverts, float *__restrict__ dscaling, float *__restrict__ drot2d) {
  extern __shared__ __align__(16) float bind_smem[];
  // thread t: face t / share of the block, its Gaussians sub, sub + share, ...
  const int t = threadIdx.x / kb.share, sub = threadIdx.x % kb.share;
  const int f0 = blockIdx.x * kb.faces, nf = min(kb.faces, b.F - f0), cap = kb.faces * kb.chunk;
  float *p = bind_smem;
  float *sq = take(p, 4 * cap), *sx = take(p, 3 * cap), *ss = take(p, 3 * cap), *s2 = take(p, 2 * cap), *r2 = take(p, 2 * cap);
  Tri T;
  bool good = true;
  float Rw[9];
  f3 g0 = mk(0.f, 0.f, 0.f), g1 = g0, g2 = g0;
  float dRw[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int gs = 0; gs < b.G; gs += kb.chunk) {  // once, unless one face's rows do not fit
    const int gn = min(kb.chunk, b.G - gs), m = nf * gn;
    const size_t o0 = (size_t)f0 * b.G + gs;
    const float *in_x = STAGED ? sx : dxyz + 3 * o0, *in_s = STAGED ? ss : dscales + 3 * o0, *in_q = STAGED ? sq : drots + 4 * o0;
    const float *in_s2 = STAGED ? s2 : b.scaling2d + 2 * o0, *in_r2 = STAGED ? r2 : b.rotation2d + 2 * o0;
    if (STAGED) {
      if (dxyz) rows_in(dxyz + 3 * o0, 3 * m, sx);
      if (dscales && dscaling) {
        rows_in(dscales + 3 * o0, 3 * m, ss);
        rows_in(b.scaling2d + 2 * o0, 2 * m, s2);
      }
      if (drots) {
        rows_in(drots + 4 * o0, 4 * m, sq);
        rows_in(b.rotation2d + 2 * o0, 2 * m, r2);
      }
    }
    if (gs == 0 && t < nf) {
      good = load_tri(b.faces, b.verts, b.V, f0 + t, T);
      if (good) {
        const Frame F = face_frame(T.v0, T.v1, T.v2);
        const float R[9] = {F.x.x, F.y.x, F.n.x, F.x.y, F.y.y, F.n.y, F.x.z, F.y.z, F.n.z};
#pragma unroll
        for (int i = 0; i < 9; ++i) Rw[i] = R[i];
      }
    }
    const bool all_good = STAGED && __syncthreads_and(good);
    if (good && t < nf) {
      for (int g = sub; g < gn; g += kb.share) {
        const int q = t * gn + g;
        if (dxyz) {
          const float *w = b.bc + 3 * (gs + g);
          const f3 d = mk(in_x[3 * q], in_x[3 * q + 1], in_x[3 * q + 2]);
          g0 = g0 + w[0] * d;
          g1 = g1 + w[1] * d;
          g2 = g2 + w[2] * d;
        }
        float ds0 = 0.f, ds1 = 0.f, dra = 0.f, drb = 0.f;
        if (dscales && dscaling) {
          ds0 = in_s[3 * q] * expf(in_s2[2 * q]);
          ds1 = in_s[3 * q + 1] * expf(in_s2[2 * q + 1]);
        }
        if (drots) {
          const float ra = in_r2[2 * q], rb = in_r2[2 * q + 1];
          const float cn = inv_norm2(ra, rb);
          const float a = ra * cn, s = rb * cn;
          float R[9];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            R[i * 3 + 0] = Rw[i * 3] * a + Rw[i * 3 + 1] * s;
            R[i * 3 + 1] = -Rw[i * 3] * s + Rw[i * 3 + 1] * a;
            R[i * 3 + 2] = Rw[i * 3 + 2];
          }
          const QuatOut qq = mat_to_quat(R);
          float dq[4];
          if (STAGED) {
            const float4 v = reinterpret_cast<const float4 *>(sq)[q];
            dq[0] = v.x; dq[1] = v.y; dq[2] = v.z; dq[3] = v.w;
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) dq[i] = in_q[4 * q + i];
          }
          float dR[9];
          mat_to_quat_adj(R, qq, dq, dR);
          float da = 0.f, ds = 0.f;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            dRw[i * 3] += dR[i * 3] * a - dR[i * 3 + 1] * s;
            dRw[i * 3 + 1] += dR[i * 3] * s + dR[i * 3 + 1] * a;
            dRw[i * 3 + 2] += dR[i * 3 + 2];
            da += dR[i * 3] * Rw[i * 3] + dR[i * 3 + 1] * Rw[i * 3 + 1];
            ds += dR[i * 3] * Rw[i * 3 + 1] - dR[i * 3 + 1] * Rw[i * 3];
          }
          // (a, s) = unit(ra, rb)
          if (cn < 1.f / NRM_EPS) {
            const float dot_ = a * da + s * ds;
            dra = (da - a * dot_) * cn;
            drb = (ds - s * dot_) * cn;
          } else {
            dra = da / NRM_EPS;
            drb = ds / NRM_EPS;
          }
        }
        if (all_good) {  // back into the rows' own places
          s2[2 * q] = ds0; s2[2 * q + 1] = ds1;
          r2[2 * q] = dra; r2[2 * q + 1] = drb;
        } else {  // a skipped face's outputs stay as the caller left them
          const size_t o = o0 + q;
          if (dscaling) { dscaling[2 * o] = ds0; dscaling[2 * o + 1] = ds1; }
          if (drot2d) { drot2d[2 * o] = dra; drot2d[2 * o + 1] = drb; }
        }
      }
    }
    if (STAGED) __syncthreads();
    if (all_good) {
      if (dscaling) rows_out(dscaling + 2 * o0, 2 * m, s2);
      if (drot2d) rows_out(drot2d + 2 * o0, 2 * m, r2);
      __syncthreads();
    }
  }
  // the face's sums over its threads
  for (int o = kb.share / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int i = 0; i < 9; ++i) dRw[i] += __shfl_xor_sync(0xffffffffu, dRw[i], o);
    g0 = g0 + shfl_xor(g0, o); g1 = g1 + shfl_xor(g1, o); g2 = g2 + shfl_xor(g2, o);
  }
  if (good && t < nf && sub == 0) {
    if (drots) {
      const Frame F = face_frame(T.v0, T.v1, T.v2);
      f3 h0, h1, h2;
      face_frame_adj(F, mk(dRw[0], dRw[3], dRw[6]), mk(dRw[1], dRw[4], dRw[7]),
                     mk(dRw[2], dRw[5], dRw[8]), h0, h1, h2);
      g0 = g0 + h0; g1 = g1 + h1; g2 = g2 + h2;
    }
    scatter_vertices(dverts, T, g0, g1, g2);
  }
}

}  // namespace

int launch_bind_fwd(const DmgsFaceBinding &b, float *xyz, float *cov, float *rot, float *covL,
                    cudaStream_t s) {
  if (b.F <= 0) return DMGS_OK;
  const FaceBlocks kb = face_blocks(b.F, b.G, 9);
  DMGS_TIMED(K_BIND_FWD, s, dmgs_host::note_launch(), bind_fwd_kernel<<<kb.blocks, BB, kb.smem, s>>>(b, kb, xyz, cov, rot, covL));
  DMGS_LAUNCH_CHECK("bind_fwd_kernel");
  return DMGS_OK;
}

int launch_bind_bwd(const DmgsFaceBinding &b, const float *dxyz, const float *dcov,
                    float *dverts, float *dsf, cudaStream_t s) {
  DMGS_CUDA(cudaMemsetAsync(dverts, 0, (size_t)b.V * 3 * 4, s));
  if (dsf) DMGS_CUDA(cudaMemsetAsync(dsf, 0, 4, s));
  if (b.F <= 0) return DMGS_OK;
  const FaceBlocks kb = face_blocks(b.F, b.G, 9);
  DMGS_TIMED(K_BIND_BWD, s, dmgs_host::note_launch(), bind_bwd_kernel<<<kb.blocks, BB, kb.smem, s>>>(b, kb, dxyz, dcov, dverts, dsf));
  DMGS_LAUNCH_CHECK("bind_bwd_kernel");
  return DMGS_OK;
}

int launch_bind3_fwd(const DmgsFaceBinding3 &b, float *xyz, float *scales, float *rots,
                     cudaStream_t s) {
  if (b.F <= 0) return DMGS_OK;
  const bool staged = b.G > DIRECT_MAX;
  const FaceBlocks kb = staged ? face_blocks(b.F, b.G, 14) : FaceBlocks{BB, b.G, (b.F - 1) / BB + 1, 1, 0};
  DMGS_TIMED(K_BIND3_FWD, s, dmgs_host::note_launch(), (staged ? bind3_fwd_kernel<true> : bind3_fwd_kernel<false>)<<<kb.blocks, BB, kb.smem, s>>>(b, kb, xyz, scales, rots));
  DMGS_LAUNCH_CHECK("bind3_fwd_kernel");
  return DMGS_OK;
}

int launch_bind3_bwd(const DmgsFaceBinding3 &b, const float *dxyz, const float *dscales,
                     const float *drots, float *dverts, float *dscaling, float *drot2d,
                     cudaStream_t s) {
  DMGS_CUDA(cudaMemsetAsync(dverts, 0, (size_t)b.V * 3 * 4, s));
  if (b.F <= 0) return DMGS_OK;
  const bool staged = b.G > DIRECT_MAX;
  const FaceBlocks kb = staged ? face_blocks(b.F, b.G, 14) : FaceBlocks{BB, b.G, (b.F - 1) / BB + 1, 1, 0};
  DMGS_TIMED(K_BIND3_BWD, s, dmgs_host::note_launch(), (staged ? bind3_bwd_kernel<true> : bind3_bwd_kernel<false>)<<<kb.blocks, BB, kb.smem, s>>>(b, kb, dxyz, dscales, drots, dverts, dscaling,
                                                     drot2d));
  DMGS_LAUNCH_CHECK("bind3_bwd_kernel");
  return DMGS_OK;
}

namespace {

constexpr int CULL_BLOCK = 256;

// Face f is in the frustum when its centroid (the mean of its vertices),
// taken through the full projection (row-vector convention of the stored
// matrix: p_j = sum_i c_i M[i][j] + M[3][j]), has |x/w|, |y/w|, |z/w| < 1.05
// with w = p_3 + 1e-6 > 0 — the stage-3 test of
// scene/gaussian_geo_model_finetune.py:33-48.  A face with a vertex index
// outside [0, V) is not kept.
__device__ __forceinline__ bool face_in_frustum(const float *__restrict__ verts, int V,
                                                const int64_t *__restrict__ faces, int f,
                                                const float *__restrict__ M) {
  int64_t vi[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    vi[k] = faces[3 * (size_t)f + k];
    if (vi[k] < 0 || vi[k] >= V) return false;
  }
  float c[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int a = 0; a < 3; ++a) c[a] += verts[3 * vi[k] + a];
#pragma unroll
  for (int a = 0; a < 3; ++a) c[a] = c[a] / 3.f;
  float p[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    p[j] = c[0] * __ldg(M + j) + c[1] * __ldg(M + 4 + j) + c[2] * __ldg(M + 8 + j) + __ldg(M + 12 + j);
  const float w = p[3] + 1e-6f;
  return w > 0.f && fabsf(p[0] / w) < 1.05f && fabsf(p[1] / w) < 1.05f && fabsf(p[2] / w) < 1.05f;
}

// The test per face, the per-block count of kept faces (for the
// order-preserving compaction).
__global__ void __launch_bounds__(CULL_BLOCK)
face_cull_test_kernel(const float *__restrict__ verts, int V, const int64_t *__restrict__ faces,
                      int F, const float *__restrict__ M, uint8_t *__restrict__ mask,
                      uint32_t *__restrict__ blkcnt) {
  const int f = blockIdx.x * CULL_BLOCK + threadIdx.x;
  const bool keep = f < F && face_in_frustum(verts, V, faces, f, M);
  if (f < F && mask) mask[f] = keep ? 1 : 0;
  const int n = __syncthreads_count(keep);
  if (threadIdx.x == 0) blkcnt[blockIdx.x] = (uint32_t)n;
}

// Kept face indices at their block's scanned offset, in face order (the
// test is recomputed: cheaper than a round trip of a flag through memory).
__global__ void __launch_bounds__(CULL_BLOCK)
face_cull_compact_kernel(const float *__restrict__ verts, int V, const int64_t *__restrict__ faces,
                         int F, const float *__restrict__ M, const uint32_t *__restrict__ blkoff,
                         int32_t *__restrict__ kept) {
  __shared__ uint32_t wcount[CULL_BLOCK / 32];
  const int f = blockIdx.x * CULL_BLOCK + threadIdx.x;
  const bool keep = f < F && face_in_frustum(verts, V, faces, f, M);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xffffffffu, keep);
  if (lane == 0) wcount[wid] = __popc(b);
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < wid; ++w) before += wcount[w];
  if (keep) {
    unsigned lt;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
    kept[blkoff[blockIdx.x] + before + __popc(b & lt)] = f;
  }
}

// Vertex frustum mask of the real-scene stage 2 (in_frustum,
// scene/gaussian_geo_model_mlp_flex_colmap.py:31-76): the grid vertex
// shifted by half a cube edge (the shift folded into the matrix's last row,
// as the reference does) taken through full_proj (row-vector convention,
// stored [4,4]); kept when w = p.w + 1e-6 > 0 and p.xyz / w lies inside the
// view's screen piece widened by 0.05 (the whole screen, a half or a
// quarter).  Optional and_mask ([N] bytes) is ANDed in.
__global__ void __launch_bounds__(256)
vertex_frustum_kernel(const float *__restrict__ verts, int N, const float *__restrict__ M, float half,
                      int piece_id, int n_piece, const uint8_t *__restrict__ and_mask,
                      uint8_t *__restrict__ out) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= N) return;
  const float x = verts[3 * (size_t)i], y = verts[3 * (size_t)i + 1], z = verts[3 * (size_t)i + 2];
  float p[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float m0 = __ldg(M + j), m1 = __ldg(M + 4 + j), m2 = __ldg(M + 8 + j);
    const float c = __fadd_rn(__ldg(M + 12 + j),
                              __fadd_rn(__fadd_rn(__fmul_rn(m0, half), __fmul_rn(m1, half)),
                                        __fmul_rn(m2, half)));
    p[j] = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, m0), __fmul_rn(y, m1)), __fmul_rn(z, m2)), c);
  }
  const float w = __fadd_rn(p[3], 1e-6f);
  const float q[3] = {__fdiv_rn(p[0], w), __fdiv_rn(p[1], w), __fdiv_rn(p[2], w)};
  bool keep;
  if (piece_id < 0) {
    keep = fabsf(q[0]) < 1.05f && fabsf(q[1]) < 1.05f && fabsf(q[2]) < 1.05f;
  } else {
    // screen piece [lo, hi] in x and y (z spans [-1, 1]), widened by 0.05
    float lx = -1.f, hx = 1.f, ly = -1.f, hy = 1.f;
    if (n_piece == 2) {
      if (piece_id == 0) hx = 0.f; else lx = 0.f;
    } else {
      if (piece_id & 1) lx = 0.f; else hx = 0.f;
      if (piece_id & 2) ly = 0.f; else hy = 0.f;
    }
    keep = q[0] > __fsub_rn(lx, 0.05f) && q[1] > __fsub_rn(ly, 0.05f) && q[2] > -1.05f &&
           q[0] < __fadd_rn(hx, 0.05f) && q[1] < __fadd_rn(hy, 0.05f) && q[2] < 1.05f;
  }
  keep = keep && w > 0.f;
  if (and_mask) keep = keep && and_mask[i] != 0;
  out[i] = keep ? 1 : 0;
}

}  // namespace

int launch_vertex_frustum(const float *verts, int N, const float *full_proj, float cube_len,
                          int piece_id, int n_piece, const uint8_t *and_mask, uint8_t *out,
                          cudaStream_t s) {
  if (N <= 0) return DMGS_OK;
  DMGS_TIMED(K_FACE_CULL, s, dmgs_host::note_launch(), vertex_frustum_kernel<<<(N + 255) / 256, 256, 0, s>>>(
      verts, N, full_proj, 0.5f * cube_len, piece_id, n_piece, and_mask, out));
  DMGS_LAUNCH_CHECK("vertex_frustum_kernel");
  return DMGS_OK;
}

size_t face_cull_scratch_bytes(int F) {
  const uint32_t nb = (uint32_t)((F + CULL_BLOCK - 1) / CULL_BLOCK);
  return align_up((size_t)nb * 4 + 4, 256) + scan_part_words(nb) * 4;
}

int launch_face_cull(const float *verts, int V, const int64_t *faces, int F,
                     const float *full_proj, uint8_t *face_mask, int32_t *kept, int32_t *num_kept,
                     char *scratch, cudaStream_t s) {
  if (F <= 0) {
    DMGS_CUDA(cudaMemsetAsync(num_kept, 0, 4, s));
    return DMGS_OK;
  }
  const uint32_t nb = (uint32_t)((F + CULL_BLOCK - 1) / CULL_BLOCK);
  uint32_t *blkcnt = reinterpret_cast<uint32_t *>(scratch);
  uint32_t *part = reinterpret_cast<uint32_t *>(scratch + align_up((size_t)nb * 4 + 4, 256));
  DMGS_TIMED(K_FACE_CULL, s, {
    dmgs_host::note_launch(), face_cull_test_kernel<<<nb, CULL_BLOCK, 0, s>>>(verts, V, faces, F, full_proj, face_mask, blkcnt);
    int r = launch_scan1(blkcnt, nb, part, reinterpret_cast<uint32_t *>(num_kept), s);
    if (r != DMGS_OK) return r;
    dmgs_host::note_launch(), face_cull_compact_kernel<<<nb, CULL_BLOCK, 0, s>>>(verts, V, faces, F, full_proj, blkcnt, kept);
  });
  DMGS_LAUNCH_CHECK("face_cull");
  return DMGS_OK;
}

}  // namespace dmgs
