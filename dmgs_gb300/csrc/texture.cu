// texture.cu — the stage-2 hash-grid texture: positions -> SH features
// (MLPTexture3D.sample_noact, geo/texture.py:101-112, called at
// scene/gaussian_geo_model_mlp_flex.py:313), forward and adjoint.
//
//   t   = clamp((xyz - lo) / (hi - lo), 0, 1)
//   enc = multiresolution hash encoding of t: 16 levels x 2 features
//         (tiny-cuda-nn HashGrid as configured at geo/texture.py:57-69:
//         base resolution 16, per-level scale 256^(1/15), 2^19 entries per
//         level, trilinear interpolation)
//   out = W3 relu(W2 relu(W1 enc))   (bias-free, geo/texture.py:18-40)
//
// Encoding conventions (Mueller et al. 2022, with tiny-cuda-nn's grid
// rules): level l has scale s_l = 2^(l log2 b) 16 - 1 and resolution
// ceil(s_l) + 1; p = t s_l + 1/2 splits into cell floor(p) and fraction;
// a corner's entry is x + y r + z r^2 while the level's dense grid fits its
// table (size r^3 rounded up to 8, capped at 2^19), else the spatial hash
// x * 1 ^ y * 2654435761 ^ z * 805459861 (32-bit), modulo the table size.
//
// Kernels:
//   forward   blocks of 128 points: a thread encodes a point (hash gathers
//             from the 50 MB table, L2-resident) into shared memory, then the
//             32-32-32-C MLP runs as register-tiled products over the block;
//   adjoint   recomputes the hidden layers from the forward's encoding, forms
//             the three weight gradients as outer-product GEMMs over the
//             block's points (each thread's entries stay in registers across
//             its tiles; one atomic per entry per block at the end) and each
//             point's dL/denc;
//   scatter   reduces the table gradient (float2 atomics, one per run of
//             consecutive points in a cell) and forms the position gradient
//             from the interpolation weights' derivatives.
// The reference's gradient hooks (geo/texture.py:72-73 with _MLP's
// loss_scale): the table receives 128x its true gradient, the positions
// their true gradient.
#include <cmath>

#include "f32x2.cuh"
#include "kernels.cuh"

namespace dmgs {

namespace {

constexpr int TEX_LEVELS = 16;
constexpr int TEX_FEAT = TEX_LEVELS * 2;  // encoding width
constexpr int TEX_THREADS = 128;
constexpr uint32_t TEX_LOG2_HASHMAP = 19;
constexpr uint32_t TEX_BASE_RES = 16;
constexpr float TEX_GRAD_SCALE = 128.f;

struct TexLevels {
  float scale[TEX_LEVELS];
  uint32_t res[TEX_LEVELS];
  uint32_t offset[TEX_LEVELS];
  uint32_t size[TEX_LEVELS];
  uint32_t hashed;  // bit l: level l is hashed
  uint32_t entries;
};

TexLevels make_levels(float per_level_scale) {
  TexLevels L{};
  // 2^(l log2 b) 16 - 1 in double from the float log2 b, rounded once
  const double log2b = (double)(float)std::log2((double)per_level_scale);
  uint32_t off = 0;
  for (int l = 0; l < TEX_LEVELS; ++l) {
    const float scale = (float)(std::exp2((double)l * log2b) * (double)TEX_BASE_RES - 1.0);
    const uint32_t res = (uint32_t)ceilf(scale) + 1u;
    const uint64_t dense = (uint64_t)res * res * res;
    const uint64_t cap = 1ull << TEX_LOG2_HASHMAP;
    const uint64_t size = std::min<uint64_t>((dense + 7) / 8 * 8, cap);
    L.scale[l] = scale;
    L.res[l] = res;
    L.offset[l] = off;
    L.size[l] = (uint32_t)size;
    if (dense > size) L.hashed |= 1u << l;
    off += (uint32_t)size;
  }
  L.entries = off;
  return L;
}

struct TexArgs {
  const float2 *table;
  const float *W1, *W2, *W3;
  float lo[3], ext[3];
  int64_t n;
};

// Entry of the corner (cx, cy, cz) of a level: the index is below twice the
// table's size on dense levels, whose tables hold every corner (the last
// plane wraps), and the hashed tables' size is a power of two.
__device__ __forceinline__ uint32_t level_entry(uint32_t cx, uint32_t cy, uint32_t cz, uint32_t res,
                                                uint32_t size, uint32_t offset, bool hashed) {
  uint32_t i;
  if (hashed) {
    i = (cx ^ (cy * 2654435761u) ^ (cz * 805459861u)) & (size - 1u);
  } else {
    i = cx + (cy + cz * res) * res;
    i = i < size ? i : i % size;
  }
  return offset + i;
}

// Normalised, clamped texture coordinate (and whether the clamp passes the
// gradient: inside [0, 1] inclusive, as torch.clamp's adjoint).
__device__ __forceinline__ void tex_coord(const TexArgs &A, const float *xyz, int64_t p, float (&t)[3],
                                          bool (&pass)[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float v = __fdiv_rn(__fsub_rn(__ldg(xyz + 3 * p + d), A.lo[d]), A.ext[d]);
    pass[d] = v >= 0.f && v <= 1.f;
    t[d] = fminf(fmaxf(v, 0.f), 1.f);
  }
}

struct LevelPos {
  uint32_t c[3];
  float f[3];
};

__device__ __forceinline__ LevelPos level_pos(const TexLevels &L, int l, const float (&t)[3]) {
  LevelPos q;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float p = __fadd_rn(__fmul_rn(t[d], L.scale[l]), 0.5f);
    const float c = floorf(p);
    q.c[d] = (uint32_t)(int)c;
    q.f[d] = __fsub_rn(p, c);
  }
  return q;
}

__device__ __forceinline__ float corner_weight(const LevelPos &q, int corner) {
  const float w0 = (corner & 1) ? q.f[0] : __fsub_rn(1.f, q.f[0]);
  const float w1 = (corner & 2) ? q.f[1] : __fsub_rn(1.f, q.f[1]);
  const float w2 = (corner & 4) ? q.f[2] : __fsub_rn(1.f, q.f[2]);
  return __fmul_rn(__fmul_rn(w0, w1), w2);
}

// ---- the block's 128 points: rows [feature][point] in shared memory -------
//
// A thread owns 8 points x TJ features of every product (points 4 pg .. + 3
// of each half of the tile, pairs of points in f32x2): per feature of the
// reduction it reads two float4 of the points' row and TJ weights for 8 TJ
// multiply-adds, where a thread per point read a weight per multiply-add and
// the kernels stood on the delivery of those broadcasts.  Every sum runs over
// the same terms in the same order as a thread per point's did.
constexpr int XP = TEX_THREADS + 4;  // row pitch: float4 rows, 8 rows start in 8 different bank groups
constexpr int WP = 36;               // weight row pitch (likewise)

struct Mine {
  int pg, jg;  // point group 0..15, feature group 0..7
  __device__ Mine() : pg(((threadIdx.x >> 6) << 3) | (threadIdx.x & 7)), jg((threadIdx.x >> 3) & 7) {}
};

// [rows][32] weights into rows of pitch WP, in flight while the block's first
// points are encoded: weights_in() before the barrier after which they are read.
// (Waited for at once they made a block of one tile slower than a thread per
// point: forward alone, 1,000 points at 48 channels, 20.5 us with a thread per
// point, 22.5 waited for, 18.5 so; 271,824 points 131, 108 and 100 us.)
__device__ __forceinline__ void load_weights(const float *__restrict__ W, int rows, float *sW) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(sW);
  for (int i = threadIdx.x; i < rows * 32; i += TEX_THREADS)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s + 4u * ((i >> 5) * WP + (i & 31))), "l"(W + i) : "memory");
}
__device__ __forceinline__ void weights_in() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The points' [n][C] rows of a tile to and from X[feature][point]: a warp
// takes 8 features of 4 points (whole 32-byte sectors; the 32 shared-memory
// words lie in 32 banks).  Points beyond n read as zero.
template <int C>
__device__ __forceinline__ void load_rows(const float *src, int64_t p0, int64_t n, float *X) {
  const int j0 = threadIdx.x & 7, q0 = threadIdx.x >> 3;
#pragma unroll
  for (int jb = 0; jb < (C + 7) / 8; ++jb)
#pragma unroll
    for (int qb = 0; qb < TEX_THREADS / 16; ++qb) {
      const int j = 8 * jb + j0, q = 16 * qb + q0;
      if (j < C) X[j * XP + q] = p0 + q < n ? src[(p0 + q) * C + j] : 0.f;
    }
}
template <int C, int POINTS, int PITCH>
__device__ __forceinline__ void store_rows(float *dst, int64_t p0, int64_t n, const float *X) {
  const int j0 = threadIdx.x & 7, q0 = threadIdx.x >> 3;
#pragma unroll
  for (int jb = 0; jb < (C + 7) / 8; ++jb)
#pragma unroll
    for (int qb = 0; qb < POINTS / 16; ++qb) {
      const int j = 8 * jb + j0, q = 16 * qb + q0;
      if (j < C && p0 + q < n) dst[(p0 + q) * C + j] = X[j * PITCH + q];
    }
}

// The encoding of the thread's point into its column of X.
__device__ __forceinline__ void encode_tile(const TexArgs &A, const TexLevels &L, const float *__restrict__ xyz,
                                            int64_t p, float *X) {
  const bool valid = p < A.n;
  float t[3] = {0.f, 0.f, 0.f};
  bool pass[3];
  if (valid) tex_coord(A, xyz, p, t, pass);
#pragma unroll 2
  for (int l = 0; l < TEX_LEVELS; ++l) {
    F2 a = f2_make(0.f, 0.f);
    if (valid) {
      const LevelPos q = level_pos(L, l, t);
      const bool hashed = (L.hashed >> l) & 1u;
      const uint32_t res = L.res[l], size = L.size[l], offset = L.offset[l];
      float2 v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c)
        v[c] = __ldg(A.table + level_entry(q.c[0] + (c & 1), q.c[1] + ((c >> 1) & 1), q.c[2] + (c >> 2), res, size,
                                           offset, hashed));
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float w = corner_weight(q, c);
        a = vadd(a, vmul(f2_make(w, w), f2_make(v[c].x, v[c].y)));
      }
    }
    X[(2 * l) * XP + threadIdx.x] = vget(a, 0);
    X[(2 * l + 1) * XP + threadIdx.x] = vget(a, 1);
  }
}

// acc[i][.] += W[j][k] X[k][points], j = jg + 8 i (rows at and beyond J are not the caller's).
template <int TJ, int J>
__device__ __forceinline__ void layer(const float *__restrict__ X, const float *__restrict__ W, const Mine &m,
                                      F2 (&acc)[TJ][4]) {
#pragma unroll
  for (int i = 0; i < TJ; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[i][q] = f2_make(0.f, 0.f);
  const float *x = X + 4 * m.pg;
  const float *w[TJ];
#pragma unroll
  for (int i = 0; i < TJ; ++i) w[i] = W + (J % 8 == 0 || m.jg + 8 * i < J ? m.jg + 8 * i : J - 1) * WP;
#pragma unroll 2
  for (int k = 0; k < 32; k += 4) {
    float4 wk[TJ];
#pragma unroll
    for (int i = 0; i < TJ; ++i) wk[i] = *reinterpret_cast<const float4 *>(w[i] + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const ulonglong2 lo = *reinterpret_cast<const ulonglong2 *>(x + (k + kk) * XP);
      const ulonglong2 hi = *reinterpret_cast<const ulonglong2 *>(x + (k + kk) * XP + TEX_THREADS / 2);
#pragma unroll
      for (int i = 0; i < TJ; ++i) {
        const float ws = kk == 0 ? wk[i].x : kk == 1 ? wk[i].y : kk == 2 ? wk[i].z : wk[i].w;
        const F2 ww = f2_make(ws, ws);
        acc[i][0] = vfma(ww, F2{lo.x}, acc[i][0]);
        acc[i][1] = vfma(ww, F2{lo.y}, acc[i][1]);
        acc[i][2] = vfma(ww, F2{hi.x}, acc[i][2]);
        acc[i][3] = vfma(ww, F2{hi.y}, acc[i][3]);
      }
    }
  }
}

__device__ __forceinline__ float4 f4_of(F2 a, F2 b) {
  return make_float4(vget(a, 0), vget(a, 1), vget(b, 0), vget(b, 1));
}

// The hidden layer's rows: relu(acc) at j = jg + 8 i.
__device__ __forceinline__ void store_relu(const F2 (&acc)[4][4], const Mine &m, float *X) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 v = f4_of(acc[i][2 * h], acc[i][2 * h + 1]);
      v.x = fmaxf(v.x, 0.f), v.y = fmaxf(v.y, 0.f), v.z = fmaxf(v.z, 0.f), v.w = fmaxf(v.w, 0.f);
      *reinterpret_cast<float4 *>(X + (m.jg + 8 * i) * XP + h * (TEX_THREADS / 2) + 4 * m.pg) = v;
    }
}

// Forward.  The encoding's gathers (the table is L2-resident) want warps in
// flight, the layers shared-memory bandwidth; blocks in different phases
// cover for each other.  271,824 points, 48 channels, float32, the encoding
// kept: 160 us with a thread per point, 119 us so (130 at five blocks an SM and
// 197 at six: the shared memory they take is L1 that the gathers lose).
template <int C>
__global__ void __launch_bounds__(TEX_THREADS, 4)
tex_fwd_kernel(const TexArgs A, const TexLevels L, const float *__restrict__ xyz, float *__restrict__ out,
               float *__restrict__ enc_out) {
  constexpr int TJ = (C + 7) / 8, SP = TEX_THREADS / 2 + 4;
  __shared__ __align__(16) float sW[(64 + C) * WP];
  __shared__ __align__(16) float X[32 * XP];  // a layer's input rows; at the end half a tile's outputs
  static_assert(8 * TJ * SP <= 32 * XP, "staged outputs fit");
  __shared__ TexLevels sL;
  float *sW1 = sW, *sW2 = sW + 32 * WP, *sW3 = sW + 64 * WP;
  if (threadIdx.x == 0) sL = L;
  load_weights(A.W1, 32, sW1);
  load_weights(A.W2, 32, sW2);
  load_weights(A.W3, C, sW3);
  const Mine m;
  const int64_t ntiles = (A.n + TEX_THREADS - 1) / TEX_THREADS;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t p0 = tile * TEX_THREADS;
    __syncthreads();  // the levels are in; the last tile's outputs are out
    encode_tile(A, sL, xyz, p0 + threadIdx.x, X);
    weights_in();
    __syncthreads();
    if (enc_out) store_rows<32, TEX_THREADS, XP>(enc_out, p0, A.n, X);  // kept for the adjoint
    {
      F2 acc[4][4];
      layer<4, 32>(X, sW1, m, acc);
      __syncthreads();
      store_relu(acc, m, X);
      __syncthreads();
      layer<4, 32>(X, sW2, m, acc);
      __syncthreads();
      store_relu(acc, m, X);
      __syncthreads();
    }
    F2 acc[TJ][4];
    layer<TJ, C>(X, sW3, m, acc);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      __syncthreads();
#pragma unroll
      for (int i = 0; i < TJ; ++i)
        *reinterpret_cast<float4 *>(X + (m.jg + 8 * i) * SP + 4 * m.pg) = f4_of(acc[i][2 * h], acc[i][2 * h + 1]);
      __syncthreads();
      store_rows<C, TEX_THREADS / 2, SP>(out, p0 + h * (TEX_THREADS / 2), A.n, X);
    }
  }
}

// acc[i][.] = sum over j of W[j][k] Y[j][points], k = 4 jg + i.
template <int J>
__device__ __forceinline__ void layer_adjoint(const float *__restrict__ Y, const float *__restrict__ W, const Mine &m,
                                              F2 (&acc)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[i][q] = f2_make(0.f, 0.f);
  const float *y = Y + 4 * m.pg, *w = W + 4 * m.jg;
#pragma unroll 4
  for (int j = 0; j < J; ++j) {
    const float4 wk = *reinterpret_cast<const float4 *>(w + j * WP);
    const ulonglong2 lo = *reinterpret_cast<const ulonglong2 *>(y + j * XP);
    const ulonglong2 hi = *reinterpret_cast<const ulonglong2 *>(y + j * XP + TEX_THREADS / 2);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float ws = i == 0 ? wk.x : i == 1 ? wk.y : i == 2 ? wk.z : wk.w;
      const F2 ww = f2_make(ws, ws);
      acc[i][0] = vfma(ww, F2{lo.x}, acc[i][0]);
      acc[i][1] = vfma(ww, F2{lo.y}, acc[i][1]);
      acc[i][2] = vfma(ww, F2{hi.x}, acc[i][2]);
      acc[i][3] = vfma(ww, F2{hi.y}, acc[i][3]);
    }
  }
}

// The rows k = 4 jg + i of H: acc where H > 0 (the layer's ReLU), else 0.
__device__ __forceinline__ void store_masked(const F2 (&acc)[4][4], const Mine &m, float *H) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 *e = reinterpret_cast<float4 *>(H + (4 * m.jg + i) * XP + h * (TEX_THREADS / 2) + 4 * m.pg);
      const float4 o = *e, d = f4_of(acc[i][2 * h], acc[i][2 * h + 1]);
      *e = make_float4(o.x > 0.f ? d.x : 0.f, o.y > 0.f ? d.y : 0.f, o.z > 0.f ? d.z : 0.f, o.w > 0.f ? d.w : 0.f);
    }
}

// A weight gradient's entries (row rg + 8 r, column cg + 8 c) over the
// points of the thread's half of the block: acc += sum over them of
// Y[row][q] X[column][q].  Rows at and beyond J are not the caller's.
template <int R, int J>
__device__ __forceinline__ void outer(const float *__restrict__ Y, const float *__restrict__ X, float (&acc)[R][4]) {
  const int half = threadIdx.x >> 6, rg = (threadIdx.x >> 3) & 7, cg = threadIdx.x & 7;
  const float *y[R], *x = X + cg * XP + half * (TEX_THREADS / 2);
#pragma unroll
  for (int r = 0; r < R; ++r)
    y[r] = Y + (J % 8 == 0 || rg + 8 * r < J ? rg + 8 * r : J - 1) * XP + half * (TEX_THREADS / 2);
#pragma unroll 2
  for (int q = 0; q < TEX_THREADS / 2; q += 4) {
    float4 xv[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) xv[c] = *reinterpret_cast<const float4 *>(x + 8 * c * XP + q);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 yv = *reinterpret_cast<const float4 *>(y[r] + q);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        acc[r][c] = fmaf(yv.x, xv[c].x, acc[r][c]);
        acc[r][c] = fmaf(yv.y, xv[c].y, acc[r][c]);
        acc[r][c] = fmaf(yv.z, xv[c].z, acc[r][c]);
        acc[r][c] = fmaf(yv.w, xv[c].w, acc[r][c]);
      }
    }
  }
}

// The block's sum of a weight gradient: the second half's entries through
// shared memory, one reduction per entry.
template <int R, int J>
__device__ __forceinline__ void reduce_outer(const float (&acc)[R][4], float *S, float *dW) {
  const int half = threadIdx.x >> 6, t = threadIdx.x & 63, rg = (threadIdx.x >> 3) & 7, cg = threadIdx.x & 7;
  __syncthreads();
  if (half)
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) S[(4 * r + c) * 64 + t] = acc[r][c];
  __syncthreads();
  if (!half)
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (J % 8 == 0 || rg + 8 * r < J)
#pragma unroll
        for (int c = 0; c < 4; ++c) atomicAdd(dW + (rg + 8 * r) * 32 + cg + 8 * c, acc[r][c] + S[(4 * r + c) * 64 + t]);
}

// Adjoint: recomputes the hidden layers, then per layer the weight gradient
// (each thread keeps its entries in registers over all its tiles) and the
// input's gradient.  Shared memory: the weights, D (the encoding, then
// dL/dout, then the encoding again), H1 and H2 (the hidden layers, each
// replaced by its own gradient).  Bound by shared-memory bandwidth; 75 KB, so
// three blocks an SM.  271,824 points, 48 channels, float32: 269 us with a
// thread per point, 150 us so (142 with the weights in flight).
constexpr size_t tex_bwd_smem(int C) {
  return (size_t)((64 + C) * WP + (C > 32 ? C : 32) * XP + 2 * 32 * XP) * sizeof(float);
}

template <int C>
__global__ void __launch_bounds__(TEX_THREADS, 3)
tex_bwd_kernel(const TexArgs A, const TexLevels L, const float *__restrict__ xyz, const float *enc_in,
               const float *__restrict__ dout, float *denc, float *__restrict__ dW1, float *__restrict__ dW2,
               float *__restrict__ dW3) {
  extern __shared__ __align__(16) float smem[];
  __shared__ TexLevels sL;
  float *sW1 = smem, *sW2 = sW1 + 32 * WP, *sW3 = sW2 + 32 * WP;
  float *H1 = sW3 + C * WP, *H2 = H1 + 32 * XP, *D = H2 + 32 * XP;
  if (threadIdx.x == 0) sL = L;
  load_weights(A.W1, 32, sW1);
  load_weights(A.W2, 32, sW2);
  load_weights(A.W3, C, sW3);
  const Mine m;
  constexpr int R3 = (C + 7) / 8;
  float acc3[R3][4], acc2[4][4], acc1[4][4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int r = 0; r < R3; ++r) acc3[r][c] = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) acc2[r][c] = acc1[r][c] = 0.f;
  }
  const float *enc = enc_in ? enc_in : denc;  // without the forward's: formed here, kept in denc's rows
  const int64_t ntiles = (A.n + TEX_THREADS - 1) / TEX_THREADS;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t p0 = tile * TEX_THREADS;
    F2 g[4][4];
    __syncthreads();  // the levels are in; the last tile's reads are done
    if (enc_in) {
      load_rows<32>(enc, p0, A.n, D);
    } else {
      encode_tile(A, sL, xyz, p0 + threadIdx.x, D);
    }
    weights_in();
    __syncthreads();
    if (!enc_in) store_rows<32, TEX_THREADS, XP>(denc, p0, A.n, D);
    layer<4, 32>(D, sW1, m, g);
    store_relu(g, m, H1);
    __syncthreads();
    load_rows<C>(dout, p0, A.n, D);
    layer<4, 32>(H1, sW2, m, g);
    store_relu(g, m, H2);
    __syncthreads();
    // layer 3: dW3 += dy h2^T;  dh2 = relu'(h2) (W3^T dy)
    outer<R3, C>(D, H2, acc3);
    layer_adjoint<C>(D, sW3, m, g);
    __syncthreads();
    store_masked(g, m, H2);
    load_rows<32>(enc, p0, A.n, D);
    __syncthreads();
    // layer 2: dW2 += dh2 h1^T;  dh1 = relu'(h1) (W2^T dh2)
    outer<4, 32>(H2, H1, acc2);
    layer_adjoint<32>(H2, sW2, m, g);
    __syncthreads();
    store_masked(g, m, H1);
    __syncthreads();
    // layer 1: dW1 += dh1 enc^T;  dL/denc = W1^T dh1
    outer<4, 32>(H1, D, acc1);
    layer_adjoint<32>(H1, sW1, m, g);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float4 *>(H2 + (4 * m.jg + i) * XP + h * (TEX_THREADS / 2) + 4 * m.pg) =
            f4_of(g[i][2 * h], g[i][2 * h + 1]);
    __syncthreads();
    store_rows<32, TEX_THREADS, XP>(denc, p0, A.n, H2);
  }
  reduce_outer<R3, C>(acc3, D, dW3);
  reduce_outer<4, 32>(acc2, D, dW2);
  reduce_outer<4, 32>(acc1, D, dW1);
}

// Table (128 x the true gradient) and position gradients from each point's
// dL/denc row: a light kernel (few registers, full occupancy) so that the
// latency of the gathers and reductions is hidden by many warps.
//
// Consecutive points lie close together (a face's Gaussians, then its
// neighbours'), so on the coarse levels most of a warp's 32 points share a
// few cells, and one reduction per point and corner hit the same few table
// entries 32 times.  Per level each lane leaves its eight corner terms and
// its cell in shared memory; lane (corner, quarter) then walks the eight
// points of its quarter in order and issues one reduction per run of equal
// cells (271,824 mesh-bound points: 366 us with a reduction per point and
// corner, 206 us so).
constexpr int SC_WARPS = 8;
constexpr int SC_PITCH = 33;  // float2s of a corner's row: eight rows start in different banks

struct ScatterSmem {
  float2 v[8][SC_PITCH];
  uint2 cell[32];      // x, y
  uint32_t cellz[32];
};

__global__ void __launch_bounds__(32 * SC_WARPS)
tex_scatter_kernel(const TexArgs A, const TexLevels L, const float *__restrict__ xyz,
                   const float *__restrict__ denc, float *__restrict__ dxyz, float2 *__restrict__ dtable) {
  __shared__ TexLevels sL;
  __shared__ ScatterSmem sm[SC_WARPS];
  if (threadIdx.x == 0) sL = L;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  ScatterSmem &S = sm[w];
  const int64_t p0 = ((int64_t)blockIdx.x * SC_WARPS + w) * 32;
  if (p0 >= A.n) return;  // warp-uniform
  const int64_t p = p0 + lane;
  const bool valid = p < A.n;
  const int nvalid = (int)(A.n - p0 < 32 ? A.n - p0 : 32);
  float t[3] = {0.f, 0.f, 0.f};
  bool pass[3] = {false, false, false};
  if (valid) tex_coord(A, xyz, p, t, pass);
  const float *dr = denc + 32 * (valid ? p : p0);
  float gt[3] = {0.f, 0.f, 0.f};
  const int corner = lane & 7, quarter = lane >> 3;
#pragma unroll 1
  for (int l = 0; l < TEX_LEVELS; ++l) {
    const LevelPos q = level_pos(sL, l, t);
    const bool hashed = (sL.hashed >> l) & 1u;
    const uint32_t res = sL.res[l], size = sL.size[l], offset = sL.offset[l];
    float2 g = *reinterpret_cast<const float2 *>(dr + 2 * l);
    if (!valid) g = make_float2(0.f, 0.f);
    float dl[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      if (dtable) {
        const float wt = corner_weight(q, c);
        S.v[c][lane] = make_float2(TEX_GRAD_SCALE * wt * g.x, TEX_GRAD_SCALE * wt * g.y);
      }
      if (dxyz) {
        const float2 v = __ldg(A.table + level_entry(q.c[0] + (c & 1), q.c[1] + ((c >> 1) & 1), q.c[2] + (c >> 2),
                                                     res, size, offset, hashed));
        const float gv = g.x * v.x + g.y * v.y;
#pragma unroll
        for (int dd = 0; dd < 3; ++dd) {
          // d w / d f_dd: the other two factors, signed by the corner's bit
          float o = 1.f;
#pragma unroll
          for (int e2 = 0; e2 < 3; ++e2)
            if (e2 != dd) o *= ((c >> e2) & 1) ? q.f[e2] : 1.f - q.f[e2];
          dl[dd] += (((c >> dd) & 1) ? o : -o) * gv;
        }
      }
    }
#pragma unroll
    for (int dd = 0; dd < 3; ++dd) gt[dd] += dl[dd] * sL.scale[l];
    if (!dtable) continue;
    S.cell[lane] = make_uint2(q.c[0], q.c[1]);
    S.cellz[lane] = q.c[2];
    __syncwarp();
    float2 sum = make_float2(0.f, 0.f);
    uint2 cell = S.cell[quarter * 8];
    uint32_t cz = S.cellz[quarter * 8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int j = quarter * 8 + i;
      const float2 v = S.v[corner][j];
      sum.x += v.x;
      sum.y += v.y;
      const uint2 next = i < 7 ? S.cell[j + 1] : cell;
      const uint32_t nz = i < 7 ? S.cellz[j + 1] : cz;
      if (i == 7 || next.x != cell.x || next.y != cell.y || nz != cz) {  // the run of this cell ends
        if (j - i < nvalid)  // a quarter beyond the last point has nothing (a run's later zeros add nothing)
          atomicAdd(dtable + level_entry(cell.x + (corner & 1), cell.y + ((corner >> 1) & 1), cz + (corner >> 2), res,
                                         size, offset, hashed),
                    sum);
        sum = make_float2(0.f, 0.f);
      }
      cell = next;
      cz = nz;
    }
    __syncwarp();  // the rows are overwritten by the next level
  }
  if (dxyz && valid)
#pragma unroll
    for (int dd = 0; dd < 3; ++dd) dxyz[3 * p + dd] = pass[dd] ? gt[dd] / A.ext[dd] : 0.f;
}

bool tex_ok(const DmgsTexture *tx) {
  if (!tx || !tx->table || !tx->W1 || !tx->W2 || !tx->W3) return false;
  if (tx->channels != 3 && tx->channels != 12 && tx->channels != 27 && tx->channels != 48) return false;
  if (!(tx->per_level_scale > 1.f)) return false;
  for (int d = 0; d < 3; ++d)
    if (!(tx->aabb[3 + d] > tx->aabb[d])) return false;
  return true;
}

TexArgs make_args(const DmgsTexture *tx, int64_t n) {
  TexArgs A;
  A.table = reinterpret_cast<const float2 *>(tx->table);
  A.W1 = tx->W1;
  A.W2 = tx->W2;
  A.W3 = tx->W3;
  for (int d = 0; d < 3; ++d) {
    A.lo[d] = tx->aabb[d];
    A.ext[d] = tx->aabb[3 + d] - tx->aabb[d];
  }
  A.n = n;
  return A;
}

// Resident blocks of a kernel, looked up once per device into the caller's
// cached_dev and cached_slots, or fewer where the points do not fill them.
template <typename K>
int persistent_grid(K kernel, size_t smem, int64_t n, int &cached_dev, int &cached_slots, int &grid) {
  int dev = 0;
  DMGS_CUDA(cudaGetDevice(&dev));
  if (dev != cached_dev) {
    int sms = 0, per = 0;
    DMGS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    DMGS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, TEX_THREADS, smem));
    cached_slots = sms * std::max(per, 1);
    cached_dev = dev;
  }
  const int64_t tiles = (n + TEX_THREADS - 1) / TEX_THREADS;
  grid = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, cached_slots));
  return DMGS_OK;
}

template <int C>
int run_fwd(const TexArgs &A, const TexLevels &L, const float *xyz, float *out, float *enc,
            cudaStream_t s) {
  thread_local int dev = -1, slots = 0;  // per channel count and host thread
  int grid;
  if (int r = persistent_grid(tex_fwd_kernel<C>, 0, A.n, dev, slots, grid)) return r;
  dmgs_host::note_launch(), tex_fwd_kernel<C><<<grid, TEX_THREADS, 0, s>>>(A, L, xyz, out, enc);
  return DMGS_OK;
}

template <int C>
int run_bwd(const TexArgs &A, const TexLevels &L, const float *xyz, const float *enc,
            const float *dout, float *dxyz, float *dtable, float *dW1, float *dW2, float *dW3,
            float *denc, cudaStream_t s) {
  if (int r = dmgs_host::raise_smem_limit((const void *)tex_bwd_kernel<C>, tex_bwd_smem(C))) return r;
  thread_local int dev = -1, slots = 0;  // per channel count and host thread
  int grid;
  if (int r = persistent_grid(tex_bwd_kernel<C>, tex_bwd_smem(C), A.n, dev, slots, grid)) return r;
  // timed apart: the MLP adjoint (weight-gradient GEMMs) and the scatter of
  // the encoding gradients into the table and the positions
  DMGS_TIMED(K_TEX_BWD, s, dmgs_host::note_launch(), tex_bwd_kernel<C><<<grid, TEX_THREADS, tex_bwd_smem(C), s>>>(
      A, L, xyz, enc, dout, denc, dW1, dW2, dW3));
  if (dxyz || dtable)
    DMGS_TIMED(K_TEX_SCATTER, s, dmgs_host::note_launch(),
               tex_scatter_kernel<<<(unsigned)((A.n + 32 * SC_WARPS - 1) / (32 * SC_WARPS)), 32 * SC_WARPS, 0, s>>>(
                   A, L, xyz, denc, dxyz, reinterpret_cast<float2 *>(dtable)));
  return DMGS_OK;
}

}  // namespace

namespace {

int tex_fwd_impl(const DmgsTexture *tx, int64_t n, const float *xyz, float *out, float *enc,
                 dmgs_stream_t stream) {
  if (!tex_ok(tx) || n < 0 || (n > 0 && (!xyz || !out)) ||
      (enc && (reinterpret_cast<uintptr_t>(enc) & 15))) {
    dmgs_host::set_error("tex_fwd: invalid arguments");
    return DMGS_ERR_ARG;
  }
  if (n == 0) return DMGS_OK;
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const TexArgs A = make_args(tx, n);
  const TexLevels L = make_levels(tx->per_level_scale);
  int r = DMGS_OK;
  DMGS_TIMED(K_TEX_FWD, s, {
    switch (tx->channels) {
      case 3: r = run_fwd<3>(A, L, xyz, out, enc, s); break;
      case 12: r = run_fwd<12>(A, L, xyz, out, enc, s); break;
      case 27: r = run_fwd<27>(A, L, xyz, out, enc, s); break;
      default: r = run_fwd<48>(A, L, xyz, out, enc, s); break;
    }
  });
  if (r != DMGS_OK) return r;
  DMGS_LAUNCH_CHECK("tex_fwd");
  return DMGS_OK;
}

int tex_bwd_impl(const DmgsTexture *tx, int64_t n, const float *xyz, const float *enc,
                 const float *dout, float *dxyz, float *dtable, float *dW1, float *dW2, float *dW3,
                 void *scratch, size_t scratch_bytes, dmgs_stream_t stream) {
  if (!tex_ok(tx) || n < 0 || !dW1 || !dW2 || !dW3 || (n > 0 && (!xyz || !dout)) ||
      (enc && (reinterpret_cast<uintptr_t>(enc) & 15))) {
    dmgs_host::set_error("tex_bwd: invalid arguments");
    return DMGS_ERR_ARG;
  }
  if (n > 0 && (!scratch || scratch_bytes < dmgs_tex_bwd_scratch_bytes(n) ||
                (reinterpret_cast<uintptr_t>(scratch) & 15))) {
    dmgs_host::set_error("tex_bwd: scratch must hold dmgs_tex_bwd_scratch_bytes(n) bytes, 16-byte aligned");
    return DMGS_ERR_STATE;
  }
  float *denc = static_cast<float *>(scratch);
  const cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const TexLevels L = make_levels(tx->per_level_scale);
  DMGS_CUDA(cudaMemsetAsync(dW1, 0, 32 * 32 * 4, s));
  DMGS_CUDA(cudaMemsetAsync(dW2, 0, 32 * 32 * 4, s));
  DMGS_CUDA(cudaMemsetAsync(dW3, 0, (size_t)tx->channels * 32 * 4, s));
  if (dtable) DMGS_CUDA(cudaMemsetAsync(dtable, 0, (size_t)L.entries * 8, s));
  if (n == 0) return DMGS_OK;
  const TexArgs A = make_args(tx, n);
  int r = DMGS_OK;
  switch (tx->channels) {
    case 3: r = run_bwd<3>(A, L, xyz, enc, dout, dxyz, dtable, dW1, dW2, dW3, denc, s); break;
    case 12: r = run_bwd<12>(A, L, xyz, enc, dout, dxyz, dtable, dW1, dW2, dW3, denc, s); break;
    case 27: r = run_bwd<27>(A, L, xyz, enc, dout, dxyz, dtable, dW1, dW2, dW3, denc, s); break;
    default: r = run_bwd<48>(A, L, xyz, enc, dout, dxyz, dtable, dW1, dW2, dW3, denc, s); break;
  }
  if (r != DMGS_OK) return r;
  DMGS_LAUNCH_CHECK("tex_bwd");
  return DMGS_OK;
}

}  // namespace

}  // namespace dmgs

using namespace dmgs;
using dmgs_host::set_error;

extern "C" {

int64_t dmgs_tex_table_entries(float per_level_scale) {
  if (!(per_level_scale > 1.f)) return -1;
  return (int64_t)make_levels(per_level_scale).entries;
}


int dmgs_tex_fwd(const DmgsTexture *tx, int64_t n, const float *xyz, float *out, dmgs_stream_t stream) {
  return tex_fwd_impl(tx, n, xyz, out, nullptr, stream);
}

int dmgs_tex_fwd_enc(const DmgsTexture *tx, int64_t n, const float *xyz, float *out, float *enc,
                     dmgs_stream_t stream) {
  if (n > 0 && !enc) {
    set_error("tex_fwd_enc: the encoding buffer is required");
    return DMGS_ERR_ARG;
  }
  return tex_fwd_impl(tx, n, xyz, out, enc, stream);
}

size_t dmgs_tex_bwd_scratch_bytes(int64_t n) { return n > 0 ? (size_t)n * 32 * sizeof(float) : 0; }

int dmgs_tex_bwd(const DmgsTexture *tx, int64_t n, const float *xyz, const float *dout, float *dxyz,
                 float *dtable, float *dW1, float *dW2, float *dW3, void *scratch,
                 size_t scratch_bytes, dmgs_stream_t stream) {
  return tex_bwd_impl(tx, n, xyz, nullptr, dout, dxyz, dtable, dW1, dW2, dW3, scratch,
                      scratch_bytes, stream);
}

int dmgs_tex_bwd_enc(const DmgsTexture *tx, int64_t n, const float *xyz, const float *enc,
                     const float *dout, float *dxyz, float *dtable, float *dW1, float *dW2,
                     float *dW3, void *scratch, size_t scratch_bytes, dmgs_stream_t stream) {
  if (n > 0 && !enc) {
    set_error("tex_bwd_enc: the encoding buffer is required");
    return DMGS_ERR_ARG;
  }
  return tex_bwd_impl(tx, n, xyz, enc, dout, dxyz, dtable, dW1, dW2, dW3, scratch, scratch_bytes,
                      stream);
}

}  // extern "C"
