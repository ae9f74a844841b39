// loss.cu — fused L1 + SSIM photometric loss and its gradient.
//
// The reference's training loss (train_geo_stage2.py:114-116 with
// utils/loss_utils.py): (1 - lambda) mean |x - y| + lambda (1 - mean SSIM),
// SSIM with an 11 x 11 Gaussian window (sigma 1.5, normalised), zero padding
// of 5, C1 = 0.01^2, C2 = 0.03^2, per channel, averaged over channels and
// pixels (Wang et al. 2004).  In torch that is five depthwise convolutions
// forward and their adjoints.  Here two kernels:
//
//   1. moments: each 32 x 54 tile of every channel loads x, y with a 5-pixel
//      halo into shared memory, blurs the five moments (x, y, xx, yy, xy)
//      separably, and per pixel forms S and the partial derivatives of S
//      w.r.t. mu_x (A), E[x^2] (B) and E[xy] (D); the block's sums of S and
//      |x - y| go to per-block partials;
//   2. gradient: each tile blurs A, B, D (the window is symmetric, so the
//      adjoint of the blur is the same blur) and forms
//      dL/dx = (1 - lambda)/N sign(x - y) - lambda/N (wA + 2 x wB + y wD);
//      the first block also reduces the partials into the loss.
//
// Bound by instruction issue: 110 multiply-adds a pixel and channel in the
// first kernel.  A thread forms four horizontal or seven vertical outputs
// from values held in registers, so that an output costs 3.5 and 2.4 shared
// loads per quantity instead of 11 (one output per thread and products kept
// in shared memory: 178 us for both kernels at 3 x 822 x 1237, against 81).
// 54 rows + 10 of halo are 64 rows of 8 groups of 4 columns (two rounds of
// the 256 threads) and 8 groups of 7 rows of 32 columns (one round); an image
// with few such tiles takes tiles of 16 rows, two vertical outputs a thread.
//
// With s11 = E[x^2] - mu_x^2, s22 = E[y^2] - mu_y^2, s12 = E[xy] - mu_x mu_y,
// N1 = 2 mu_x mu_y + C1, N2 = 2 s12 + C2, D1 = mu_x^2 + mu_y^2 + C1,
// D2 = s11 + s22 + C2, S = N1 N2 / (D1 D2):
//   dS/dE[x^2] = -S / D2,  dS/dE[xy] = 2 N1 / (D1 D2),
//   dS/dmu_x   = 2 mu_y (N2 - N1) / (D1 D2) - 2 mu_x S / D1 + 2 mu_x S / D2.
#include <cmath>

#include "kernels.cuh"

namespace dmgs {

namespace {

constexpr int LR = 5;              // window radius
constexpr int LTAP = 2 * LR + 1;
constexpr int LW = 32;             // columns of an output tile
constexpr int LP = 44;             // pitch of a haloed row (42 columns; rows 16-byte aligned)
constexpr int LN = 256;            // threads

// A tile whose threads form LV vertical outputs each.
template <int LV>
struct Tile {
  static constexpr int LHT = LV == 7 ? 54 : LV * (LN / LW);  // output rows
  static constexpr int LROWS = LHT + 2 * LR;                 // rows with the halo
  static constexpr int LHS = LV * (LN / LW) + 2 * LR;        // rows the vertical pass reads (of 7: the last two of no output)
};
static_assert(Tile<7>::LROWS * (LW / 4) == 2 * LN && LW * ((Tile<7>::LHT + 6) / 7) == LN, "tile and block sizes");

struct Window {
  float w[LTAP];
};

// One or two images' haloed tile into shared memory, zero outside the image:
// a warp per row (columns lane and lane + 32), rows LN / 32 apart, so that a
// row's bounds are the warp's and no index is divided.
template <int LROWS, int NQ>
__device__ __forceinline__ void load_tile(const float *__restrict__ a, const float *__restrict__ b, int H, int Wd,
                                          int ox, int oy, float (*da)[LP], float (*db)[LP]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int x0 = ox + lane, x1 = x0 + 32;
  const bool in0 = x0 >= 0 && x0 < Wd, more = lane < LW + 2 * LR - 32, in1 = more && x1 < Wd;
#pragma unroll 4
  for (int r = w; r < LROWS; r += LN / 32) {
    const int gy = oy + r;
    const bool row = gy >= 0 && gy < H;
    const size_t o = (size_t)(row ? gy : 0) * Wd;
    const float a0 = row && in0 ? a[o + x0] : 0.f, a1 = row && in1 ? a[o + x1] : 0.f;
    float b0 = 0.f, b1 = 0.f;
    if (NQ == 2) {
      b0 = row && in0 ? b[o + x0] : 0.f;
      b1 = row && in1 ? b[o + x1] : 0.f;
    }
    da[r][lane] = a0;
    if (more) da[r][lane + 32] = a1;
    if (NQ == 2) {
      db[r][lane] = b0;
      if (more) db[r][lane + 32] = b1;
    }
  }
}

// Row r's 14 values from column 4 g on.
__device__ __forceinline__ void load_row(const float (*src)[LP], int r, int g, float (&v)[16]) {
  const float4 *p = reinterpret_cast<const float4 *>(&src[r][4 * g]);
#pragma unroll
  for (int k = 0; k < 4; ++k) {  // the last two of the 16 (of the pitch's padding at most) are not used
    const float4 x = p[k];
    v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
  }
}

// Four horizontal outputs of a quantity, taps in ascending order.
__device__ __forceinline__ float4 blur4(const Window &W, const float (&v)[16]) {
  float o[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < LTAP; ++k) a = fmaf(W.w[k], v[j + k], a);
    o[j] = a;
  }
  return make_float4(o[0], o[1], o[2], o[3]);
}

// The thread's LV vertical outputs of a quantity (column c, rows LV gv ..).
template <int LV>
__device__ __forceinline__ void blur_column(const Window &W, const float (*hs)[LW], int c, int gv, float (&o)[LV]) {
  float v[LV + 2 * LR];
#pragma unroll
  for (int k = 0; k < LV + 2 * LR; ++k) v[k] = hs[gv * LV + k][c];
#pragma unroll
  for (int j = 0; j < LV; ++j) {
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < LTAP; ++k) a = fmaf(W.w[k], v[j + k], a);
    o[j] = a;
  }
}

__device__ __forceinline__ float block_sum(float v, float *red) {
  const int t = threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((t & 31) == 0) red[t >> 5] = v;
  __syncthreads();
  float s = 0.f;
  if (t < LN / 32) s = red[t];
  if (t < 32) {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return s;  // valid in thread 0
}

template <int LV>
struct MomentsSmem {
  float x[Tile<LV>::LROWS][LP], y[Tile<LV>::LROWS][LP];
  float hs[5][Tile<LV>::LHS][LW];
  float red[LN / 32];
};

template <int LV>
struct GradSmem {
  float in[Tile<LV>::LROWS][LP];
  float hs[3][Tile<LV>::LHS][LW];
  float red[LN / 32];
};

// Grid: (tiles x, tiles y, channels).  ABD: [3][C][H][W] scratch;
// part: 2 floats per block (sum S, sum |x - y|).
template <int LV>
__global__ void __launch_bounds__(LN)
ssim_moments_kernel(const float *__restrict__ x, const float *__restrict__ y, int H, int Wd,
                    Window W, float *__restrict__ ABD, float *__restrict__ part) {
  extern __shared__ __align__(16) char loss_smem[];
  constexpr int LHT = Tile<LV>::LHT, LROWS = Tile<LV>::LROWS;
  MomentsSmem<LV> &sm = *reinterpret_cast<MomentsSmem<LV> *>(loss_smem);
  const int c = blockIdx.z, t = threadIdx.x;
  const size_t plane = (size_t)H * Wd;
  const int ox = blockIdx.x * LW, oy = blockIdx.y * LHT;
  load_tile<LROWS, 2>(x + c * plane, y + c * plane, H, Wd, ox - LR, oy - LR, sm.x, sm.y);
  __syncthreads();
#pragma unroll 1
  for (int i = t; i < LROWS * (LW / 4); i += LN) {
    const int r = i >> 3, g = i & 7;
    float a[16], b[16], p[16];
    load_row(sm.x, r, g, a);
    load_row(sm.y, r, g, b);
    auto put = [&](int q, float4 v) { *reinterpret_cast<float4 *>(&sm.hs[q][r][4 * g]) = v; };
    put(0, blur4(W, a));
    put(1, blur4(W, b));
#pragma unroll
    for (int k = 0; k < 14; ++k) p[k] = __fmul_rn(a[k], a[k]);
    put(2, blur4(W, p));
#pragma unroll
    for (int k = 0; k < 14; ++k) p[k] = __fmul_rn(b[k], b[k]);
    put(3, blur4(W, p));
#pragma unroll
    for (int k = 0; k < 14; ++k) p[k] = __fmul_rn(a[k], b[k]);
    put(4, blur4(W, p));
  }
  __syncthreads();
  const int col = t & (LW - 1), gv = t / LW;
  float m[5][LV];
#pragma unroll
  for (int q = 0; q < 5; ++q) blur_column<LV>(W, sm.hs[q], col, gv, m[q]);
  float S_sum = 0.f, l1 = 0.f;
  const int px = ox + col;
#pragma unroll
  for (int j = 0; j < LV; ++j) {
    const int row = gv * LV + j, py = oy + row;
    if (row >= LHT || px >= Wd || py >= H) continue;
    constexpr float C1 = 0.01f * 0.01f, C2 = 0.03f * 0.03f;
    const float mx = m[0][j], my = m[1][j];
    const float s11 = m[2][j] - mx * mx, s22 = m[3][j] - my * my, s12 = m[4][j] - mx * my;
    const float N1 = 2.f * mx * my + C1, N2 = 2.f * s12 + C2;
    const float D1 = mx * mx + my * my + C1, D2 = s11 + s22 + C2;
    const float inv = 1.f / (D1 * D2);
    const float S = N1 * N2 * inv;
    // S / D1, S / D2; S is 0 where D1 or D2 has overflowed (inv is 0), and inf * 0 would be NaN
    const float S1 = S == 0.f ? 0.f : S * (D2 * inv), S2 = S == 0.f ? 0.f : S * (D1 * inv);
    const float A = 2.f * my * (N2 - N1) * inv - 2.f * mx * S1 + 2.f * mx * S2;
    const float B = -S2;
    const float Dd = 2.f * N1 * inv;
    const size_t o = c * plane + (size_t)py * Wd + px;
    const size_t all = (size_t)gridDim.z * plane;
    ABD[o] = A;
    ABD[all + o] = B;
    ABD[2 * all + o] = Dd;
    S_sum += S;
    l1 += fabsf(sm.x[row + LR][col + LR] - sm.y[row + LR][col + LR]);
  }
  const float sS = block_sum(S_sum, sm.red);
  __syncthreads();
  const float sL = block_sum(l1, sm.red);
  if (t == 0) {
    const size_t b = ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    part[2 * b] = sS;
    part[2 * b + 1] = sL;
  }
}

template <int LV>
__global__ void __launch_bounds__(LN)
ssim_grad_kernel(const float *__restrict__ x, const float *__restrict__ y, int H, int Wd,
                 Window W, const float *__restrict__ ABD, float lambda, float inv_n,
                 float *__restrict__ grad, const float *__restrict__ part, int nparts,
                 float *__restrict__ loss) {
  extern __shared__ __align__(16) char loss_smem[];
  constexpr int LHT = Tile<LV>::LHT, LROWS = Tile<LV>::LROWS;
  GradSmem<LV> &sm = *reinterpret_cast<GradSmem<LV> *>(loss_smem);
  const int c = blockIdx.z, t = threadIdx.x;
  const size_t plane = (size_t)H * Wd;
  const size_t all = (size_t)gridDim.z * plane;
  const int ox = blockIdx.x * LW, oy = blockIdx.y * LHT;
#pragma unroll 1
  for (int q = 0; q < 3; ++q) {
    load_tile<LROWS, 1>(ABD + q * all + c * plane, nullptr, H, Wd, ox - LR, oy - LR, sm.in, nullptr);
    __syncthreads();
#pragma unroll
    for (int i = t; i < LROWS * (LW / 4); i += LN) {
      const int r = i >> 3, g = i & 7;
      float a[16];
      load_row(sm.in, r, g, a);
      *reinterpret_cast<float4 *>(&sm.hs[q][r][4 * g]) = blur4(W, a);
    }
    __syncthreads();
  }
  const int col = t & (LW - 1), gv = t / LW;
  float b[3][LV];
#pragma unroll
  for (int q = 0; q < 3; ++q) blur_column<LV>(W, sm.hs[q], col, gv, b[q]);
  const int px = ox + col;
#pragma unroll
  for (int j = 0; j < LV; ++j) {
    const int row = gv * LV + j, py = oy + row;
    if (row >= LHT || px >= Wd || py >= H) continue;
    const size_t o = c * plane + (size_t)py * Wd + px;
    const float xv = x[o], yv = y[o], d = xv - yv;
    const float sgn = (d > 0.f) ? 1.f : (d < 0.f ? -1.f : 0.f);
    const float dS = b[0][j] + 2.f * xv * b[1][j] + yv * b[2][j];
    grad[o] = (1.f - lambda) * inv_n * sgn - lambda * inv_n * dS;
  }
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && loss) {
    // the partials of all blocks of the moments kernel (launched before)
    float sS = 0.f, sL = 0.f;
    for (int i = t; i < nparts; i += LN) {
      sS += part[2 * i];
      sL += part[2 * i + 1];
    }
    __syncthreads();
    sS = block_sum(sS, sm.red);
    __syncthreads();
    sL = block_sum(sL, sm.red);
    if (t == 0) *loss = (1.f - lambda) * sL * inv_n + lambda * (1.f - sS * inv_n);
  }
}

Window gaussian_window() {
  Window W;
  double g[2 * LR + 1], sum = 0.0;
  for (int k = -LR; k <= LR; ++k) {
    g[k + LR] = std::exp(-(double)(k * k) / (2.0 * 1.5 * 1.5));
    sum += g[k + LR];
  }
  for (int k = 0; k <= 2 * LR; ++k) W.w[k] = (float)(g[k] / sum);
  return W;
}

size_t tiles(int C, int H, int W, int rows) {
  return (size_t)C * ((H + rows - 1) / rows) * ((W + LW - 1) / LW);
}

// The small tile (LV = 2, 16 rows) where there are fewer than two large ones per
// SM: the large one has too few blocks there, and a thread forms its seven
// outputs one after the other.  Both kernels, 3 channels, large | small tile:
// 128 x 128 20.6 | 18.4 us, 256 x 256 20.5 | 20.6, 320 x 320 24.7 | 22.6,
// 400 x 400 28.7 | 28.7, 512 x 512 35.0 | 36.6 (LV = 1: 18.5, 23.2, 26.8, 35.0,
// 48.2; LV = 4: 20.5, 21.8, 23.0, 28.7, 36.3).
constexpr int LSMALL = 2;
bool small_tiles(int C, int H, int W) { return tiles(C, H, W, Tile<7>::LHT) < 2 * (size_t)NUM_SMS_HINT; }

size_t nblocks(int C, int H, int W) {
  return tiles(C, H, W, small_tiles(C, H, W) ? Tile<LSMALL>::LHT : Tile<7>::LHT);
}

template <int LV>
int run(const float *x, const float *y, int C, int H, int W, float lambda, float *loss, float *grad, float *ABD, float *part,
        cudaStream_t s) {
  const Window win = gaussian_window();
  const dim3 grid((W + LW - 1) / LW, (H + Tile<LV>::LHT - 1) / Tile<LV>::LHT, C);
  const size_t m_smem = sizeof(MomentsSmem<LV>), g_smem = sizeof(GradSmem<LV>);
  if (int r = dmgs_host::raise_smem_limit((const void *)ssim_moments_kernel<LV>, m_smem)) return r;
  if (int r = dmgs_host::raise_smem_limit((const void *)ssim_grad_kernel<LV>, g_smem)) return r;
  const float inv_n = 1.f / ((float)C * (float)H * (float)W);
  DMGS_TIMED(K_LOSS, s, {
    dmgs_host::note_launch(), ssim_moments_kernel<LV><<<grid, LN, m_smem, s>>>(x, y, H, W, win, ABD, part);
    dmgs_host::note_launch(), ssim_grad_kernel<LV><<<grid, LN, g_smem, s>>>(
        x, y, H, W, win, ABD, lambda, inv_n, grad, part, (int)(grid.x * grid.y * grid.z), loss);
  });
  DMGS_LAUNCH_CHECK("ssim kernels");
  return DMGS_OK;
}

}  // namespace

}  // namespace dmgs

using namespace dmgs;

extern "C" size_t dmgs_l1_ssim_scratch_bytes(int32_t C, int32_t H, int32_t W) {
  if (C <= 0 || H <= 0 || W <= 0) return 0;
  return l1_ssim_scratch_bytes(C, H, W);
}

extern "C" int dmgs_l1_ssim(const float *image, const float *target, int32_t C, int32_t H,
                            int32_t W, float lambda_dssim, float *loss, float *grad, void *scratch,
                            size_t scratch_bytes, dmgs_stream_t stream) {
  if (C <= 0 || H <= 0 || W <= 0 || !image || !target || !grad) {
    dmgs_host::set_error("l1_ssim: invalid arguments");
    return DMGS_ERR_ARG;
  }
  if (!scratch || scratch_bytes < l1_ssim_scratch_bytes(C, H, W)) {
    dmgs_host::set_error("l1_ssim: scratch too small");
    return DMGS_ERR_STATE;
  }
  return launch_l1_ssim(image, target, C, H, W, lambda_dssim, loss, grad,
                        static_cast<char *>(scratch), reinterpret_cast<cudaStream_t>(stream));
}

namespace dmgs {

size_t l1_ssim_scratch_bytes(int C, int H, int W) {
  return align_up((size_t)3 * C * H * W * 4, 256) + nblocks(C, H, W) * 8;
}

int launch_l1_ssim(const float *x, const float *y, int C, int H, int W, float lambda,
                   float *loss, float *grad, char *scratch, cudaStream_t s) {
  float *ABD = reinterpret_cast<float *>(scratch);
  float *part = reinterpret_cast<float *>(scratch + align_up((size_t)3 * C * H * W * 4, 256));
  return small_tiles(C, H, W) ? run<LSMALL>(x, y, C, H, W, lambda, loss, grad, ABD, part, s)
                              : run<7>(x, y, C, H, W, lambda, loss, grad, ABD, part, s);
}

}  // namespace dmgs
