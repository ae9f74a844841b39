// blend_warp.cu — the default form of the blend forward and adjoint: every
// warp blends its own part of a tile, from a work list sorted by cost.
//
// Semantics and per-pixel arithmetic are those of blend.cu (the tunable
// CTA-per-tile form); images are bit-identical.  What differs:
// * the unit of work is a part of a tile for one warp: a half (16 x 8
//   pixels, 4 per lane) or, where the tile's list is long against what every
//   warp has to do, a strip (16 x 2 pixels, one per lane).  No block
//   barriers: a warp stages 32 list entries at a time, keeps those whose
//   footprint meets its own rows, and ends when its own pixels are done;
// * parts are taken from a queue in descending order of the tiles' list
//   lengths (the ranges kernel sorts them into half-octave classes), so that
//   no long tile starts last, and strips keep one long tile from being the
//   whole launch: a list is a serial chain.  Splitting every tile is no gain:
//   a wide footprint then visits four times the warps;
// * a lane's pixels are held as packed pairs and their arithmetic issued as
//   f32x2 instructions (same roundings): the kernels are bound by issue.
#include <algorithm>

#include "blend_common.cuh"
#include "f32x2.cuh"

namespace dmgs {

namespace {

constexpr int BW_WARPS = 2;  // warps per CTA (independent of one another)

// A lane's PPT pixels: G groups of N.
template <int PPT>
struct Px;
template <>
struct Px<1> {
  static constexpr int N = 1, G = 1;
  using V = float;
  static __device__ __forceinline__ V splat(float x) { return x; }
  static __device__ __forceinline__ V make(const float *x) { return x[0]; }
  static __device__ __forceinline__ float sum(V x) { return x; }
};
template <int PPT>
struct Px {
  static constexpr int N = 2, G = PPT / 2;
  using V = F2;
  static __device__ __forceinline__ V splat(float x) { return f2_make(x, x); }
  static __device__ __forceinline__ V make(const float *x) { return f2_make(x[0], x[1]); }
  static __device__ __forceinline__ float sum(V x) { return vget(x, 0) + vget(x, 1); }
};

// ---- staging ------------------------------------------------------------------

// Whether a Gaussian's alpha can reach 1/255 in tile columns 0-15 and rows
// r0 .. r0 + RB - 1 of the tile at (ox, oy): a superset of what the per-pixel
// test accepts.  (A, B, C) is the conic scaled for ex2, thr = log2(1/(255 o));
// the exponent A dx^2 + B dx dy + C dy^2 is concave for a definite conic.
// RB = 2: each row's maximum (dx = k dy clamped to the columns); else the
// maximum over the rectangle: 0 when it holds the centre, otherwise on one of
// the four edges, each the 1D maximum clamped to its edge.  The ranges are
// widened by 0.01 pixels and the threshold lowered by 0.01 + 1e-5 x the
// largest magnitude of the terms, far above the rounding of either evaluation.
template <int RB>
__device__ __forceinline__ bool band_hit(float a, float b, float c, float o, float A, float B,
                                         float C, float thr, float cx, float cy, float r0) {
  if (!(o >= ALPHA_MIN)) return false;  // alpha <= o < 1/255 everywhere
  if (!(a * c - b * b > 0.f) || !(a > 0.f) || !(c > 0.f) || !(A < 0.f) || !(C < 0.f))
    return true;  // not an ellipse
  const float lo = cx - 15.01f, hi = cx + 0.01f;
  const float X = fmaxf(fabsf(lo), fabsf(hi)), Y = fmaxf(fabsf(cy), fabsf(cy - 15.f));
  const float mag = fabsf(A) * X * X + fabsf(B) * X * Y + fabsf(C) * Y * Y;
  const float lim = thr - (0.01f + 1e-5f * mag);
  const float kx = __fdividef(-0.5f * B, A);
  auto ev = [&](float dx, float dy) { return fmaf(fmaf(C, dy, B * dx), dy, A * dx * dx); };
  auto row = [&](float dy) { return ev(fminf(fmaxf(kx * dy, lo), hi), dy); };
  if (RB == 2) return row(cy - r0) >= lim || row(cy - r0 - 1.f) >= lim;
  const float ylo = cy - (r0 + (float)(RB - 1)) - 0.01f, yhi = cy - r0 + 0.01f;
  const float ky = __fdividef(-0.5f * B, C);
  float e = fmaxf(row(ylo), row(yhi));
  e = fmaxf(e, ev(lo, fminf(fmaxf(ky * lo, ylo), yhi)));
  e = fmaxf(e, ev(hi, fminf(fmaxf(ky * hi, ylo), yhi)));
  return e >= lim || (lo <= 0.f && hi >= 0.f && ylo <= 0.f && yhi >= 0.f);
}

// A staged Gaussian in shared memory: what every lane reads per visit, three
// 16-byte words.  (Storing the factors of packed products twice, so that they
// arrive as register pairs, took five words: a broadcast load still delivers
// its bytes to every lane, and the forward went from 1.87 to 2.05 ms for 16
// views of 3M Gaussians.)
struct Entry {
  float x, y, A, B, C, o, thr, r, g, b;
  uint32_t pos;
  __device__ __forceinline__ void put(float4 (*S)[32], int s) const {
    S[0][s] = make_float4(x, y, A, B);
    S[1][s] = make_float4(C, o, thr, __uint_as_float(pos));
    S[2][s] = make_float4(r, g, b, 0.f);
  }
  __device__ __forceinline__ void get(const float4 (*S)[32], int s) {
    const float4 a = S[0][s], c = S[1][s], d = S[2][s];
    x = a.x; y = a.y; A = a.z; B = a.w; C = c.x; o = c.y; thr = c.z; pos = __float_as_uint(c.w);
    r = d.x; g = d.y; b = d.z;
  }
};

// ---- work items ---------------------------------------------------------------

struct Item {
  int view, tile, part;
  bool fine;
};

// Smallest list length of class c (BLEND_CLASSES - 1: empty lists).
__device__ __forceinline__ uint32_t class_floor(int c) {
  if (c >= BLEND_CLASSES - 1) return 0u;
  const int b = BLEND_CLASSES - 2 - c, l = b >> 1;
  return (b & 1) && l > 0 ? 3u << (l - 1) : 1u << l;
}

// A tile is split into strips when its list is at least this share of the
// list entries a warp walks on average.
constexpr float FINE_SHARE = 1.0f;
constexpr int PARTS_FINE = 8, PARTS_COARSE = 2;

struct WorkTable {
  uint32_t first[MAX_BATCH_VIEWS * BLEND_CLASSES];  // exclusive prefix of the items, view-major
  uint32_t total;
  uint32_t shares;      // parts in which the adjoint clears its spans
  uint32_t fine_floor;  // lists of classes whose floor is at least this are split into strips
};

// Built once per CTA (all threads); ctas: those that the tiles can feed.
template <bool SKIP_EMPTY>
__device__ __forceinline__ void build_table(const BlendWork &wk, int nviews, unsigned ctas, WorkTable &tab) {
  const int tid = threadIdx.x, n = nviews * BLEND_CLASSES;
  if (tid < 32) {
    float k = tid < nviews ? (float)wk.v[tid].counters[CI_K] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(FULL, k, o);
    const float share = FINE_SHARE * k * PARTS_COARSE / (float)(ctas * BW_WARPS);
    if (tid == 0) tab.fine_floor = (uint32_t)fminf(fmaxf(share, 1.f), 4e9f);
  }
  __syncthreads();
  const uint32_t ff = tab.fine_floor;
  for (int i = tid; i < n; i += 32 * BW_WARPS) {
    const int v = i / BLEND_CLASSES, c = i % BLEND_CLASSES;
    const uint32_t parts = SKIP_EMPTY && c == BLEND_CLASSES - 1 ? 0u
                           : class_floor(c) >= ff               ? PARTS_FINE
                                                                : PARTS_COARSE;
    tab.first[i] = wk.v[v].cls_n[c] * parts;
  }
  __syncthreads();
  if (tid < 32) {
    constexpr int PER = MAX_BATCH_VIEWS * BLEND_CLASSES / 32;
    uint32_t sum = 0;
    for (int k = 0; k < PER; ++k) sum += tid * PER + k < n ? tab.first[tid * PER + k] : 0u;
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(FULL, incl, o);
      if (tid >= o) incl += u;
    }
    if (tid == 31) tab.total = incl;
    uint32_t run = incl - sum;
    for (int k = 0; k < PER; ++k)
      if (tid * PER + k < n) {
        const uint32_t x = tab.first[tid * PER + k];
        tab.first[tid * PER + k] = run;
        run += x;
      }
  }
  __syncthreads();
}

// Item i (i < total), found by the whole warp.
__device__ __forceinline__ Item find_item(const BlendWork &wk, const BlendBatch &bb, const WorkTable &tab,
                                          uint32_t i, int lane) {
  constexpr int PER = MAX_BATCH_VIEWS * BLEND_CLASSES / 32;
  const int n = bb.nviews * BLEND_CLASSES;
  // the last entry whose first item is <= i (empty entries share their successor's)
  const bool c1 = lane * PER < n && tab.first[lane * PER] <= i;
  const int b = 31 - __clz(__ballot_sync(FULL, c1));
  const int q = b * PER + lane;
  const bool c2 = lane < PER && q < n && tab.first[q] <= i;
  const int e = b * PER + 31 - __clz(__ballot_sync(FULL, c2));
  Item it;
  it.view = e / BLEND_CLASSES;
  const int c = e % BLEND_CLASSES;
  it.fine = class_floor(c) >= tab.fine_floor;
  const uint32_t k = i - tab.first[e], parts = it.fine ? PARTS_FINE : PARTS_COARSE;
  it.part = (int)(k % parts);
  it.tile = (int)wk.v[it.view].cls_list[class_slot(c, k / parts, bb.v[it.view].T)];
  return it;
}

__device__ __forceinline__ uint32_t take_item(uint32_t *queue, int lane) {
  uint32_t i = 0;
  if (lane == 0) i = atomicAdd(queue, 1u);
  return __shfl_sync(FULL, i, 0);
}

// ---- forward --------------------------------------------------------------------

template <int PPT>
__device__ __forceinline__ void fwd_part(const BlendView &V, int tile, int part, float4 (*S)[32], int lane) {
  using P = Px<PPT>;
  using F = typename P::V;
  constexpr int RB = 2 * PPT, N = P::N, G = P::G;
  const int tx = tile % V.gx, ty = tile / V.gx;
  const int px = tx * TILE + (lane & 15), py0 = ty * TILE + part * RB + (lane >> 4);
  const float pxf = (float)px, ox = (float)(tx * TILE), oy = (float)(ty * TILE), r0 = (float)(part * RB);
  const uint2 range = V.ranges[tile];
  const uint32_t n = range.y - range.x;
  const uint32_t *__restrict__ list = V.point_list + range.x;
  bool done[PPT];
  uint32_t last[PPT];
  F npy[G], T[G], cr[G], cg[G], cb[G];
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float y[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int k = g * N + i, py = py0 + 2 * k;
      done[k] = !(px < V.W && py < V.H);
      last[k] = 0u;
      y[i] = -(float)py;
    }
    npy[g] = P::make(y);
    T[g] = P::splat(1.f);
    cr[g] = cg[g] = cb[g] = P::splat(0.f);
  }
  auto all_done = [&]() {
    bool d = true;
#pragma unroll
    for (int k = 0; k < PPT; ++k) d = d && done[k];
    return __all_sync(FULL, d);
  };
  const F one = P::splat(1.f), minus = P::splat(-1.f);
  float4 f0, f1, f2;
  uint32_t id = (uint32_t)lane < n ? list[lane] : 0xffffffffu;
  load_record(V, id, f0, f1, f2);
  id = 32u + lane < n ? list[32 + lane] : 0xffffffffu;
  for (uint32_t base = 0; base < n; base += 32) {
    if (all_done()) break;
    // stage the entries that can reach this part's rows, in list order
    const float A = __fmul_rn(-0.5f * LOG2E, f0.z), B = __fmul_rn(-LOG2E, f0.w), C = __fmul_rn(-0.5f * LOG2E, f1.x);
    const float thr = -LOG2_255 - __log2f(f1.y);
    const bool hit = base + lane < n &&
                     band_hit<RB>(f0.z, f0.w, f1.x, f1.y, A, B, C, thr, f0.x - ox, f0.y - oy, r0);
    const unsigned bal = __ballot_sync(FULL, hit);
    if (hit) {
      const Entry E{f0.x, f0.y, A, B, C, f1.y, thr, f1.z, f1.w, f2.x, base + lane + 1u};
      E.put(S, __popc(bal & lanemask_lt()));
    }
    // the next entries' records and the indices after them, in flight meanwhile
    if (base + 32 < n) {
      load_record(V, id, f0, f1, f2);
      id = base + 64u + lane < n ? list[base + 64 + lane] : 0xffffffffu;
    }
    __syncwarp();
    const int nv = __popc(bal);
    for (int i = 0; i < nv; ++i) {
      Entry E;
      E.get(S, i);
      const float dx = __fsub_rn(E.x, pxf);
      const F ax2 = P::splat(__fmul_rn(__fmul_rn(E.A, dx), dx)), q = P::splat(__fmul_rn(E.B, dx));
      float e[PPT];
      bool ok[PPT], any = false;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const F dy = vadd(P::splat(E.y), npy[g]);
        const F ee = vfma(vfma(P::splat(E.C), dy, q), dy, ax2);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int k = g * N + j;
          e[k] = vget(ee, j);
          ok[k] = !done[k] && !(e[k] > 0.f) && !(e[k] < E.thr);
          any |= ok[k];
        }
      }
      if (!__any_sync(FULL, any)) continue;  // warp-uniform
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float al[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int k = g * N + j;
          const float a = fminf(ALPHA_MAX, __fmul_rn(E.o, ex2_approx(e[k])));
          al[j] = ok[k] && !(a < ALPHA_MIN) ? a : 0.f;
        }
        const F tT = vmul(T[g], vfma(P::make(al), minus, one));  // T where alpha is 0
        float nT[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int k = g * N + j;
          const float t = vget(tT, j);
          const bool stop = t < T_EPS;  // a pixel that is not done has T >= T_EPS
          nT[j] = stop ? vget(T[g], j) : t;
          al[j] = stop ? 0.f : al[j];
          done[k] = done[k] || stop;
          last[k] = al[j] > 0.f ? E.pos : last[k];
        }
        const F w = vmul(P::make(al), T[g]);
        T[g] = P::make(nT);
        cr[g] = vfma(P::splat(E.r), w, cr[g]);
        cg[g] = vfma(P::splat(E.g), w, cg[g]);
        cb[g] = vfma(P::splat(E.b), w, cb[g]);
      }
    }
    __syncwarp();  // the staged entries are overwritten by the next batch
  }
  const size_t HW = (size_t)V.H * V.W;
  const float bgr = __ldg(V.bg), bgg = __ldg(V.bg + 1), bgb = __ldg(V.bg + 2);
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const int py = py0 + 2 * k;
    if (!(px < V.W && py < V.H)) continue;
    const int pix = py * V.W + px;
    const float t = vget(T[k / N], k % N);
    V.final_T[pix] = t;
    V.n_contrib[pix] = last[k];
    V.out_color[pix] = vget(cr[k / N], k % N) + t * bgr;
    V.out_color[HW + pix] = vget(cg[k / N], k % N) + t * bgg;
    V.out_color[2 * HW + pix] = vget(cb[k / N], k % N) + t * bgb;
  }
}

__global__ void __launch_bounds__(32 * BW_WARPS)
blend_fwd_warp_kernel(const BlendBatch bb, const BlendWork wk, uint32_t *queue) {
  __shared__ WorkTable tab;
  __shared__ float4 S[BW_WARPS][3][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  build_table<false>(wk, bb.nviews, gridDim.x, tab);
  for (uint32_t i = take_item(queue, lane); i < tab.total; i = take_item(queue, lane)) {
    const Item it = find_item(wk, bb, tab, i, lane);
    const BlendView &V = bb.v[it.view];
    if (it.fine) fwd_part<1>(V, it.tile, it.part, S[w], lane);
    else fwd_part<4>(V, it.tile, it.part, S[w], lane);
  }
}

// ---- adjoint --------------------------------------------------------------------

// What the warp's visits leave to be summed over its lanes: per Gaussian nine
// rows of 32 (with Gd = dL/dopacity's term of a pixel: dL/dndc x and y per
// unit opacity, sums of Gd dx^2, Gd dx dy, Gd dy^2, Gd, and of dL/drgb),
// RED_N Gaussians at a time.  Lane t < 9 RED_N then adds up row t (16-byte
// loads; the pitch puts eight consecutive rows in different banks) and issues
// one reduction: 20 instructions a Gaussian, where a shuffle tree per visit
// took 48.  The NDC terms a dx + b dy and b dx + c dy are formed per lane:
// for a needle the two products nearly cancel, and summed apart first their
// rounding would be that of the whole sums.
constexpr int RED_N = 3, RED_P = 36;

struct alignas(16) Pending {
  float row[9 * RED_N][RED_P];
  float opacity[RED_N];
  uint32_t id[RED_N];
};

__device__ __forceinline__ void flush_pending(Pending &R, int n, float *gacc, int lane) {
  __syncwarp();
  if (lane < 9 * n) {
    const float4 *r = reinterpret_cast<const float4 *>(R.row[lane]);
    // lanes 16, 8, 4, 2, 1 apart in turn: the rounding of a shuffle tree
    auto add = [](float4 x, float4 y) { return make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w); };
    const float4 a = add(add(add(r[0], r[4]), add(r[2], r[6])), add(add(r[1], r[5]), add(r[3], r[7])));
    const int which = lane / 9, slot = lane - 9 * which;
    float v = (a.x + a.z) + (a.y + a.w);
    if (slot < 5) v *= R.opacity[which];  // dL/dpower = o Gd
    if (slot >= 2 && slot < 5) v *= slot == 3 ? -1.f : -0.5f;  // the conic's terms
    atomicAdd(gacc + (size_t)R.id[which] * 12 + slot, v);
  }
  __syncwarp();
}

// SAFE selects a pixel's terms where they otherwise are scaled by 0, which is
// not 0 for what is not finite: with a NaN in one pixel's gradient only the
// Gaussians blended there are to see it.  The plain form leaves a part with
// such a gradient (or one whose products could overflow) to the other, and
// returns false (16 views of 1M Gaussians: 2363 us; 2554 with the selections in
// every part's loop).
template <int PPT, bool SAFE>
__device__ __forceinline__ bool bwd_part(const BlendView &V, int tile, int part, float4 (*S)[32], float4 *K,
                                         uint32_t *I, Pending &R, int lane) {
  using P = Px<PPT>;
  using F = typename P::V;
  constexpr int RB = 2 * PPT, N = P::N, G = P::G;
  const int tx = tile % V.gx, ty = tile / V.gx;
  const int px = tx * TILE + (lane & 15), py0 = ty * TILE + part * RB + (lane >> 4);
  const float pxf = (float)px, ox = (float)(tx * TILE), oy = (float)(ty * TILE), r0 = (float)(part * RB);
  const uint2 range = V.ranges[tile];
  const uint32_t *__restrict__ list = V.point_list + range.x;
  const size_t HW = (size_t)V.H * V.W;
  const float bg0 = __ldg(V.bg), bg1 = __ldg(V.bg + 1), bg2 = __ldg(V.bg + 2);
  // per pixel: transmittance, -T_final (bg . dL/dpixel), dL/dpixel, and the
  // colour accumulated behind the visited Gaussian dotted with dL/dpixel
  F npy[G], T[G], nTfb[G], g0[G], g1[G], g2[G], ag[G];
  uint32_t last[PPT], most = 0u;
  bool odd = false;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    float y[N], t[N], b[N], d0[N], d1[N], d2[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int k = g * N + j, py = py0 + 2 * k;
      const bool in = px < V.W && py < V.H;
      const size_t pix = (size_t)py * V.W + px;
      y[j] = -(float)py;
      t[j] = in ? V.final_T[pix] : 0.f;
      last[k] = in ? V.n_contrib[pix] : 0u;
      d0[j] = in ? V.dL_dout[pix] : 0.f;
      d1[j] = in ? V.dL_dout[HW + pix] : 0.f;
      d2[j] = in ? V.dL_dout[2 * HW + pix] : 0.f;
      b[j] = -(t[j] * (bg0 * d0[j] + bg1 * d1[j] + bg2 * d2[j]));
      most = max(most, last[k]);
      odd = odd || !(fabsf(d0[j]) + fabsf(d1[j]) + fabsf(d2[j]) + fabsf(b[j]) < 1e18f);
    }
    npy[g] = P::make(y); T[g] = P::make(t); nTfb[g] = P::make(b);
    g0[g] = P::make(d0); g1[g] = P::make(d1); g2[g] = P::make(d2);
    ag[g] = P::splat(0.f);
  }
  if (!SAFE && __any_sync(FULL, odd)) return false;
  most = __reduce_max_sync(FULL, most);
  most = min(most, range.y - range.x);  // list positions from `most` on are never blended
  const float hw = 0.5f * (float)V.W, hh = 0.5f * (float)V.H;
  const F minus = P::splat(-1.f);
  // back to front: entry `most - 1 - j` for j = 0, 1, ...
  auto entry = [&](uint32_t j) { return j < most ? list[most - 1u - j] : 0xffffffffu; };
  int np = 0;  // Gaussians pending in R
  float4 f0, f1, f2;
  uint32_t id = entry(lane), nid = entry(32u + lane);
  load_record(V, id, f0, f1, f2);
  for (uint32_t base = 0; base < most; base += 32) {
    const float A = __fmul_rn(-0.5f * LOG2E, f0.z), B = __fmul_rn(-LOG2E, f0.w), C = __fmul_rn(-0.5f * LOG2E, f1.x);
    const float thr = -LOG2_255 - __log2f(f1.y);
    const bool hit = base + lane < most && id < V.P &&
                     band_hit<RB>(f0.z, f0.w, f1.x, f1.y, A, B, C, thr, f0.x - ox, f0.y - oy, r0);
    const unsigned bal = __ballot_sync(FULL, hit);
    if (hit) {
      const int s = __popc(bal & lanemask_lt());
      const Entry E{f0.x, f0.y, A, B, C, f1.y, thr, f1.z, f1.w, f2.x, most - 1u - base - lane};
      E.put(S, s);
      K[s] = make_float4(-f0.z * hw, -f0.w * hw, -f1.x * hh, -f0.w * hh);
      I[s] = id;
    }
    if (base + 32 < most) {
      id = nid;
      load_record(V, id, f0, f1, f2);
      nid = entry(base + 64u + lane);
    }
    __syncwarp();
    const int nv = __popc(bal);
    for (int i = 0; i < nv; ++i) {
      Entry E;
      E.get(S, i);
      const float dx = __fsub_rn(E.x, pxf);
      const F ax2 = P::splat(__fmul_rn(__fmul_rn(E.A, dx), dx)), q = P::splat(__fmul_rn(E.B, dx));
      float e2[PPT];
      bool ok[PPT], any = false;
      F dy[G];
#pragma unroll
      for (int g = 0; g < G; ++g) {
        dy[g] = vadd(P::splat(E.y), npy[g]);
        const F ee = vfma(vfma(P::splat(E.C), dy[g], q), dy[g], ax2);
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int k = g * N + j;
          e2[k] = vget(ee, j);
          ok[k] = E.pos < last[k] && !(e2[k] > 0.f) && !(e2[k] < E.thr);
          any |= ok[k];
        }
      }
      if (!__any_sync(FULL, any)) continue;  // warp-uniform
      F M[6];  // sums of Gd, Gd dy, Gd dy^2, and of dL/drgb, over the lane's pixel groups
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float G_[N], al[N], iv[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int k = g * N + j;
          const float ex = ex2_approx(e2[k]);
          const float a = fminf(ALPHA_MAX, __fmul_rn(E.o, ex));
          const bool take = ok[k] && !(a < ALPHA_MIN);
          al[j] = take ? a : 0.f;
          G_[j] = take ? ex : 0.f;
          iv[j] = take ? rcp_approx(1.f - a) : 1.f;  // T stays as it is
        }
        const F inv = P::make(iv), at = P::make(al);
        const F Tn = vmul(T[g], inv);
        const F cdg = vfma(P::splat(E.b), g2[g], vfma(P::splat(E.g), g1[g], vmul(P::splat(E.r), g0[g])));
        const F Sd = vfma(ag[g], minus, cdg);  // (c - acc) . dL/dpixel
        const F dLa = vfma(Sd, Tn, vmul(nTfb[g], inv));
        F Gd = vmul(P::make(G_), dLa);         // dL/dopacity term
        if (SAFE) {  // al is 0 where the Gaussian is not blended
          float gd[N];
#pragma unroll
          for (int j = 0; j < N; ++j) gd[j] = al[j] > 0.f ? vget(Gd, j) : 0.f;
          Gd = P::make(gd);
        }
        const F wt = vmul(at, Tn);             // dL/drgb weight
        const F gy = vmul(Gd, dy[g]);
        T[g] = Tn;
        ag[g] = vfma(at, Sd, ag[g]);
        if (g == 0) {
          M[0] = Gd; M[1] = gy; M[2] = vmul(gy, dy[g]);
          M[3] = vmul(wt, g0[g]); M[4] = vmul(wt, g1[g]); M[5] = vmul(wt, g2[g]);
        } else {
          M[0] = vadd(M[0], Gd); M[1] = vadd(M[1], gy); M[2] = vfma(gy, dy[g], M[2]);
          M[3] = vfma(wt, g0[g], M[3]); M[4] = vfma(wt, g1[g], M[4]); M[5] = vfma(wt, g2[g], M[5]);
        }
      }
      // the lane's pixels share dx
      const float m0 = P::sum(M[0]), m1 = P::sum(M[1]), mx = dx * m0;
      float(*row)[RED_P] = R.row + 9 * np;
      const float4 kk = K[i];
      row[0][lane] = mx * kk.x + m1 * kk.y;
      row[1][lane] = m1 * kk.z + mx * kk.w;
      row[2][lane] = mx * dx;
      row[3][lane] = m1 * dx;
      row[4][lane] = P::sum(M[2]);
      row[5][lane] = m0;
      row[6][lane] = P::sum(M[3]);
      row[7][lane] = P::sum(M[4]);
      row[8][lane] = P::sum(M[5]);
      if (lane == 0) {
        R.opacity[np] = E.o;
        R.id[np] = I[i];
      }
      if (++np == RED_N) {
        flush_pending(R, RED_N, V.gacc, lane);
        np = 0;
      }
    }
    __syncwarp();
  }
  if (np > 0) flush_pending(R, np, V.gacc, lane);
  return true;
}

__global__ void __launch_bounds__(32 * BW_WARPS, 10)
blend_bwd_warp_kernel(const BlendBatch bb, const BlendWork wk, const ZeroSpans zero, unsigned ctas, uint32_t *queue) {
  __shared__ WorkTable tab;
  __shared__ float4 S[BW_WARPS][3][32];
  __shared__ float4 K[BW_WARPS][32];
  __shared__ uint32_t I[BW_WARPS][32];
  __shared__ Pending R[BW_WARPS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  build_table<true>(wk, bb.nviews, ctas, tab);
  // The spans are cleared a share per item, spread over the launch (all at its
  // start they took as long as alone: 0.11 ms for 744 MB); where there are
  // fewer items than warps, a share per warp, the last ones by warps that no
  // item is left for: 3M Gaussians in a view of one tile took 7.5 ms with a
  // share to each of eight items, 1.8 ms so.  (The number of shares is kept in
  // shared memory: a register more through the loop cost 5%.)
  if (threadIdx.x == 0) tab.shares = max(tab.total, gridDim.x * BW_WARPS);
  __syncthreads();
  uint32_t i = take_item(queue, lane);
  for (; i < tab.total; i = take_item(queue, lane)) {
    const Item it = find_item(wk, bb, tab, i, lane);
    const BlendView &V = bb.v[it.view];
    zero_spans(zero, i, tab.shares, lane, 32u);
    const bool done = it.fine ? bwd_part<1, false>(V, it.tile, it.part, S[w], K[w], I[w], R[w], lane)
                              : bwd_part<4, false>(V, it.tile, it.part, S[w], K[w], I[w], R[w], lane);
    if (!done) {  // rare: strips alone, a half being four of them
      const int n = it.fine ? 1 : 4;
#pragma unroll 1
      for (int p = 0; p < n; ++p) bwd_part<1, true>(V, it.tile, n * it.part + p, S[w], K[w], I[w], R[w], lane);
    }
  }
  if (zero.n == 0) return;
  for (; i < tab.shares; i = take_item(queue, lane)) zero_spans(zero, i, tab.shares, lane, 32u);
}

// Resident CTAs of a kernel (looked up once per device and host thread), at
// most what `total` tiles can feed.
template <typename K>
int resident_grid(K kernel, int total, int &dev_, int &slots_, int &grid) {
  int dev = 0;
  DMGS_CUDA(cudaGetDevice(&dev));
  if (dev != dev_) {
    int sms = 0, per = 0;
    DMGS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    DMGS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 32 * BW_WARPS, 0));
    slots_ = sms * max(per, 1);
    dev_ = dev;
  }
  grid = (int)std::max(1ll, std::min((long long)slots_, (long long)total * PARTS_FINE / BW_WARPS));
  return DMGS_OK;
}

}  // namespace

int launch_blend_warp_fwd(const BlendBatch &bb, const BlendWork &wk, uint32_t *queue, cudaStream_t s) {
  thread_local int dev = -1, slots = 0;
  int grid;
  if (int r = resident_grid(blend_fwd_warp_kernel, bb.total, dev, slots, grid)) return r;
  DMGS_TIMED(K_BLEND_FWD, s, dmgs_host::note_launch(), blend_fwd_warp_kernel<<<grid, 32 * BW_WARPS, 0, s>>>(bb, wk, queue));
  DMGS_LAUNCH_CHECK("blend_fwd_warp_kernel");
  return DMGS_OK;
}

int launch_blend_warp_bwd(const BlendBatch &bb, const BlendWork &wk, const ZeroSpans &zero, uint32_t *queue,
                          cudaStream_t s) {
  thread_local int dev = -1, slots = 0;
  int ctas;
  if (int r = resident_grid(blend_bwd_warp_kernel, bb.total, dev, slots, ctas)) return r;
  // more CTAs than the tiles feed where there is enough to clear: 16 KB a warp
  size_t words = 0;
  for (int k = 0; k < zero.n; ++k) words += zero.words[k];
  const int grid = std::max(ctas, (int)std::min<size_t>(slots, words / (4096 * BW_WARPS) + 1));
  DMGS_TIMED(K_BLEND_BWD, s, dmgs_host::note_launch(), blend_bwd_warp_kernel<<<grid, 32 * BW_WARPS, 0, s>>>(bb, wk, zero, ctas, queue));
  DMGS_LAUNCH_CHECK("blend_bwd_warp_kernel");
  return DMGS_OK;
}

}  // namespace dmgs
