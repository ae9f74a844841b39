// binning.cu — (tile, Gaussian) lists ordered by depth, without sorting the
// instance list.
//
// The reference pipeline (duplicateWithKeys -> radix sort of the 64-bit
// (tile << 32 | depth_bits) instance keys -> identifyTileRanges) yields, per
// tile, the covering Gaussians in depth order, ties in Gaussian-index order.
// The same lists are produced here with work linear in the visible Gaussians
// V, their (Gaussian, tile row) pairs K1 and the instances K:
//
//   1. compact   the visible Gaussians in index order: (depth_bits, index);
//   2. sort      them by depth bits with a stable LSD radix sort (4 x 8-bit
//                digits) -> depth order, ties in index order;
//   3. chunk     the sorted list is cut into C contiguous chunks of equal
//                work (weight of a Gaussian: CHUNK_W_GAUSS + its tile rows
//                / 16 + its tiles / 64) -> chunk starts; the packed tile rectangles are laid
//                out in sorted order on the way (srect);
//   4. rows      each chunk counts its Gaussians per tile row (a 1D
//                difference array) -> row counts [gy][C], scanned flat into
//                the offsets of the ROW LISTS: per tile row, the Gaussians
//                covering it in depth order, each entry {index, x0 | x1 << 16};
//   5. segments  groups of C / S consecutive chunks (row segments) count
//                their instances per tile (a 2D difference grid over a band
//                of tile rows) -> segment counts [T][S], scanned flat into
//                every (tile, segment)'s list offset, K and the tile ranges;
//   6. emit      one warp per chunk appends its Gaussians to the row lists
//                (the rows of its Gaussians spread over the lanes, ranks of
//                equal rows by bitwise ballots); then one block per (tile row,
//                segment) splits that segment of the row list into its
//                tiles' lists through a shared-memory staging buffer (counts,
//                offsets and ranks per sub-pass) and copies each tile's run
//                out contiguously.
//
// Every step keeps depth order within a tile: chunks and segments are depth
// ranges laid out in depth order, and within a warp the instances are ranked
// in Gaussian order.  Nothing of size K is sorted or read back; the K-sized
// list is written once, in runs, and the row lists (K1 8-byte entries) are
// written once and read once.  The row and segment offsets are small (gy x C
// and T x S words).
//
// Launches: steps 1-5 are nine kernels (compaction, four sort passes, chunks,
// counts, scans, ranges), step 6 two.  Every prefix that crosses blocks is formed by
// decoupled look-back inside the kernel that needs it, so no step has a scan
// launch of its own and the sort reads its keys once per pass: a view has
// 10^4-10^6 visible Gaussians, a few us of memory traffic, and its time was
// launches (41 of them: 0.21 ms per view at 3M Gaussians, 0.14M visible).
//
// Every kernel bins several views at once (one grid dimension, each view with
// its own geometry state and sizes): a batch of views fills the GPU with one
// launch per stage instead of one small launch per stage and view.  In the
// look-back kernels the view is the fast grid dimension: the tiles that start
// together then belong to all views and have few predecessors each.
#include <algorithm>
#include <cmath>

#include "kernels.cuh"

namespace dmgs {

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Block-wide exclusive scan of one value per thread (u64 accumulation).
template <int THREADS>
__device__ __forceinline__ unsigned long long block_exclusive_scan(unsigned long long v,
                                                                   unsigned long long *total) {
  __shared__ unsigned long long warp_sums[THREADS / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  unsigned long long inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long u = __shfl_up_sync(FULL, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) warp_sums[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    unsigned long long s = lane < THREADS / 32 ? warp_sums[lane] : 0ull;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(FULL, s, o);
      if (lane >= o) s += u;
    }
    if (lane < THREADS / 32) warp_sums[lane] = s;  // inclusive
  }
  __syncthreads();
  const unsigned long long before = (wid > 0 ? warp_sums[wid - 1] : 0ull) + inc - v;
  if (total) *total = warp_sums[THREADS / 32 - 1];
  __syncthreads();
  return before;
}

// ---- generic exclusive scan (u32, in place), three phases ------------------

__global__ void __launch_bounds__(SCAN_THREADS)
scan_reduce_kernel(const uint32_t *__restrict__ data, uint32_t n, uint32_t *__restrict__ part) {
  for (uint32_t tile = blockIdx.x; tile * (uint32_t)SCAN_TILE < n; tile += gridDim.x) {
    const uint32_t base = tile * SCAN_TILE;
    unsigned long long s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
      const uint32_t k = base + i * SCAN_THREADS + threadIdx.x;
      if (k < n) s += data[k];
    }
    unsigned long long tot;
    block_exclusive_scan<SCAN_THREADS>(s, &tot);
    if (threadIdx.x == 0) part[tile] = (uint32_t)tot;
  }
}

// One block: exclusive scan of the per-block partials (or of the whole array
// when it fits one block); total to *total_out.
__global__ void __launch_bounds__(SCAN_THREADS)
scan_single_kernel(uint32_t *__restrict__ data, uint32_t n, uint32_t *__restrict__ total_out) {
  const uint32_t per = (n + SCAN_THREADS - 1) / SCAN_THREADS;
  const uint32_t beg = min(n, threadIdx.x * per), end = min(n, beg + per);
  unsigned long long s = 0;
  for (uint32_t k = beg; k < end; ++k) s += data[k];
  unsigned long long tot;
  unsigned long long run = block_exclusive_scan<SCAN_THREADS>(s, &tot);
  for (uint32_t k = beg; k < end; ++k) {
    const uint32_t x = data[k];
    data[k] = (uint32_t)run;
    run += x;
  }
  if (threadIdx.x == 0 && total_out) *total_out = (uint32_t)tot;
}

__global__ void __launch_bounds__(SCAN_THREADS)
scan_down_kernel(uint32_t *__restrict__ data, uint32_t n, const uint32_t *__restrict__ part) {
  for (uint32_t tile = blockIdx.x; tile * (uint32_t)SCAN_TILE < n; tile += gridDim.x) {
    // blocked: thread i owns elements base + i*ITEMS .. +ITEMS-1
    uint32_t x[SCAN_ITEMS];
    unsigned long long s = 0;
    const uint32_t k0 = tile * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
      x[i] = (k0 + i < n) ? data[k0 + i] : 0u;
      s += x[i];
    }
    unsigned long long run = block_exclusive_scan<SCAN_THREADS>(s, nullptr) + part[tile];
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; ++i) {
      if (k0 + i < n) data[k0 + i] = (uint32_t)run;
      run += x[i];
    }
  }
}

// ---- decoupled look-back ---------------------------------------------------
//
// Blocks take their tile from a ticket counter, so every predecessor of a
// tile is held by a block that runs already and never waits for a later one.
// A tile publishes its aggregate, adds up its predecessors' words back to one
// that holds an inclusive prefix, and publishes its own.  Each word carries
// its state in its top two bits and is written whole, so relaxed accesses
// suffice.  The polls are bounded: a tile that gives up (or sees that another
// has) sets ST_BOUNDS and ST_WAIT, and every later kernel then leaves the view
// alone.

constexpr unsigned long long LB_AGG = 1ull << 62, LB_INC = 2ull << 62, LB_VAL = LB_AGG - 1;
constexpr uint32_t LB32_AGG = 1u << 30, LB32_INC = 2u << 30, LB32_VAL = LB32_AGG - 1;
#ifndef DMGS_LB_POLLS
#define DMGS_LB_POLLS (1u << 20)  // about a second
#endif
constexpr uint32_t LB_POLLS = DMGS_LB_POLLS;
constexpr uint32_t ST_GAVE_UP = ST_BOUNDS | ST_WAIT;

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long *p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t *p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(unsigned long long *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

constexpr uint32_t ST_STOP = ST_OVERFLOW | ST_BOUNDS;  // a view no later binning kernel touches

__device__ __forceinline__ bool give_up(uint32_t polls, const uint32_t *counters) {
  return polls > LB_POLLS || ((polls & 255u) == 255u && (ld_relaxed(counters + CI_STATUS) & ST_BOUNDS));
}

// Exclusive prefix of `agg` at tile t, called by one whole warp; *ok is false
// when the wait was given up.
__device__ __forceinline__ unsigned long long lookback(unsigned long long *st, uint32_t t,
                                                       unsigned long long agg,
                                                       const uint32_t *counters, bool *ok) {
  const int lane = threadIdx.x & 31;
  *ok = true;
  if (lane == 0) st_relaxed(st + t, (t == 0 ? LB_INC : LB_AGG) | agg);
  if (t == 0) return 0ull;
  unsigned long long excl = 0;
  long long base = (long long)t - 1;
  for (uint32_t polls = 0;;) {
    const long long i = base - lane;
    const unsigned long long w = i >= 0 ? ld_relaxed(st + i) : LB_INC;
    const uint32_t state = (uint32_t)(w >> 62);
    const unsigned inc = __ballot_sync(FULL, state == 2u), none = __ballot_sync(FULL, state == 0u);
    const int last = inc ? __ffs(inc) - 1 : 31;  // words of lanes 0..last are added
    if (none & (0xffffffffu >> (31 - last))) {
      // one decision for the warp: its lanes' loads of the status may differ
      if (__any_sync(FULL, give_up(++polls, counters))) {
        *ok = false;
        return 0ull;
      }
      continue;
    }
    unsigned long long v = lane <= last ? w & LB_VAL : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    excl += v;
    if (inc) break;
    base -= 32;
  }
  if (lane == 0) st_relaxed(st + t, LB_INC | (excl + agg));
  return excl;
}

// Whether the view is one to leave alone: the same answer for all threads of
// the block, also while another block of this launch sets the bit.
__device__ __forceinline__ bool stopped(const BinView &B) {
  return __syncthreads_or((B.counters[CI_STATUS] & ST_STOP) != 0u);
}

// Next tile of this block (the same for all its threads).
__device__ __forceinline__ uint32_t take_ticket(uint32_t *ticket, uint32_t *slot) {
  __syncthreads();
  if (threadIdx.x == 0) *slot = atomicAdd(ticket, 1u);
  __syncthreads();
  return *slot;
}

// Chunks of a view with V visible Gaussians.
__device__ __forceinline__ uint32_t chunk_count(const BinView &B, uint32_t V) {
  return min((V + CHUNK_MIN_GAUSS - 1) / CHUNK_MIN_GAUSS, B.cmax);
}

// rect = (x0 | y0 << 16, x1 | y1 << 16): tiles [x0, x1) x [y0, y1)
__device__ __forceinline__ void unpack_rect(uint2 r, int &x0, int &y0, int &x1, int &y1) {
  x0 = (int)(r.x & 0xffffu); y0 = (int)(r.x >> 16); x1 = (int)(r.y & 0xffffu); y1 = (int)(r.y >> 16);
}

// The work a Gaussian costs the binning kernels: a fixed part, one per 16
// covered tile rows for the row lists and one per 64 covered tiles for the
// tile lists.
__device__ __forceinline__ uint32_t chunk_weight(uint2 r) {
  int x0, y0, x1, y1;
  unpack_rect(r, x0, y0, x1, y1);
  const uint32_t rows = (uint32_t)(y1 - y0), area = rows * (uint32_t)(x1 - x0);
  return CHUNK_W_GAUSS + (rows + 15u) / 16u + (area + 63u) / 64u;
}

// ---- steps 1, 2: compaction of the visible Gaussians, radix sort ------------

// One block per RADIX_TILE Gaussians, CPT consecutive per thread (their flag
// bytes read as one word): the visible ones in index order, as (depth bits,
// index) for the sort and as the list the adjoint walks, from the position
// that the preprocess's counts give the tile (the earlier groups' sums and
// the earlier tiles of its own group).  On the way: the
// digit histograms of all four sort passes, the total chunk weight, and the
// zeros of the sort's look-back words (a tile's share; the tiles the sort
// uses are at most those here).
constexpr int CPT = RADIX_TILE / PRE_BLOCK;
static_assert(VGROUP <= 32, "a group's tiles are summed by one warp");
static_assert(CPT == 8, "the flag bytes of a thread are read as one 8-byte word");

__global__ void __launch_bounds__(PRE_BLOCK)
compact_kernel(const BinViews bv) {
  const BinView &B = bv.v[blockIdx.x];
  __shared__ uint32_t hist[4 * 256], wsum[PRE_BLOCK / 32], wweight[PRE_BLOCK / 32];
  __shared__ uint32_t s_excl;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  for (uint32_t tile = blockIdx.y; tile < (uint32_t)B.nb_radix; tile += gridDim.y) {
#pragma unroll
    for (int p = 0; p < 4; ++p) hist[p * 256 + tid] = 0u;
#pragma unroll
    for (int p = 0; p < 4; ++p) B.stsort[((size_t)p * B.nb_radix + tile) * 256 + tid] = 0u;
    const int i0 = (int)tile * RADIX_TILE + tid * CPT;
    uint2 f8 = make_uint2(0u, 0u);
    if (i0 + CPT <= B.P) {
      f8 = *reinterpret_cast<const uint2 *>(B.flags + i0);  // i0 % 8 == 0, the array 256-byte aligned
    } else {
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (i0 + k < B.P) (k < 4 ? f8.x : f8.y) |= (uint32_t)B.flags[i0 + k] << (8 * (k & 3));
    }
    uint32_t vis = 0u;
#pragma unroll
    for (int k = 0; k < CPT; ++k)
      vis |= (((k < 4 ? f8.x : f8.y) >> (8 * (k & 3))) & FLAG_VISIBLE) ? 1u << k : 0u;
    const uint32_t c = __popc(vis);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    uint32_t before = incl - c, total = 0u;
#pragma unroll
    for (int w = 0; w < PRE_BLOCK / 32; ++w) {
      before += w < wid ? wsum[w] : 0u;
      total += wsum[w];
    }
    // depth and rectangle of the visible ones (the record's third float4)
    uint32_t key[CPT], weight = 0u;
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      key[k] = 0u;
      if ((vis >> k) & 1u) {
        const float4 f2 = B.feat[3 * (size_t)(i0 + k) + 2];
        key[k] = __float_as_uint(f2.y);
        weight += chunk_weight(make_uint2(__float_as_uint(f2.z), __float_as_uint(f2.w)));
      }
    }
    if (wid == 0) {
      const uint32_t group = tile / VGROUP;
      uint32_t e = lane < tile % VGROUP ? B.vtile[group * VGROUP + lane] : 0u;
      for (uint32_t g = lane; g < group; g += 32) e += B.vgroup[g];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(FULL, e, o);
      if (lane == 0) {
        s_excl = e;
        if (tile == (uint32_t)B.nb_radix - 1) B.counters[CI_V] = e + total;
      }
    }
#pragma unroll
    for (int k = 0; k < CPT; ++k)
      if ((vis >> k) & 1u)
#pragma unroll
        for (int p = 0; p < 4; ++p) atomicAdd(&hist[p * 256 + ((key[k] >> (8 * p)) & 255u)], 1u);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) weight += __shfl_xor_sync(FULL, weight, o);
    if (lane == 0) wweight[wid] = weight;
    __syncthreads();
    uint32_t pos = s_excl + before;
#pragma unroll
    for (int k = 0; k < CPT; ++k)
      if ((vis >> k) & 1u) {
        B.k0[pos] = key[k];
        B.v0[pos] = (uint32_t)(i0 + k);
        B.vlist[pos] = (uint32_t)(i0 + k);
        ++pos;
      }
    if (tid == 0) {
      unsigned long long w = 0;
#pragma unroll
      for (int i = 0; i < PRE_BLOCK / 32; ++i) w += wweight[i];
      if (w) atomicAdd(reinterpret_cast<unsigned long long *>(B.counters + CI_W), w);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const uint32_t h = hist[p * 256 + tid];
      if (h) atomicAdd(&B.ghist[p * 256 + tid], h);
    }
    __syncthreads();  // hist and the sums are cleared for the next tile
  }
}

// Lanes whose 8-bit digit equals this lane's (invalid lanes, digit 256, group
// together): nine ballots instead of match.any.
__device__ __forceinline__ unsigned digit_peers(int d) {
  unsigned peers = FULL;
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    const bool bit = (d >> b) & 1;
    const unsigned m = __ballot_sync(FULL, bit);
    peers &= bit ? m : ~m;
  }
  return peers;
}

// One pass of the stable LSD sort of (depth bits, index) by 8-bit digits:
// every block counts its tile's digits, thread d looks back over the earlier
// tiles' counts of digit d (LB_WIDE words at a time: the first wave's tiles
// all start together, and their chain would otherwise cost one memory
// latency per tile; four passes over 0.14M keys of one view / 3.5M of 16
// took 42 / 232 us at 4 words, 50 / 206 at 8, 43 / 284 at 16, and 115 / 280
// as separate histogram, scan and scatter launches), and the tile is
// scattered to its final place.  Warp w
// of a tile owns keys [w*256, +256), visited in 8 rounds of 32 (round-major,
// then lane) — the input order, so the pass is stable.
constexpr int LB_WIDE = 4;

__global__ void __launch_bounds__(RADIX_BLOCK)
radix_pass_kernel(const BinViews bv, int pass) {
  const BinView &B = bv.v[blockIdx.x];
  // pass p reads (k0, v0) when p is even and writes (k1, v1), and back
  const uint32_t *kin = (pass & 1) ? B.k1 : B.k0, *vin = (pass & 1) ? B.v1 : B.v0;
  uint32_t *kout = (pass & 1) ? B.k0 : B.k1, *vout = (pass & 1) ? B.v0 : B.v1;
  const int shift = 8 * pass;
  const uint32_t V = B.counters[CI_V], ntiles = (V + RADIX_TILE - 1) / RADIX_TILE;
  if (blockIdx.y >= ntiles || stopped(B)) return;
  __shared__ uint32_t wh[RADIX_BLOCK / 32][256];
  __shared__ uint32_t slot, wsum[RADIX_BLOCK / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  // digit tid's first position: exclusive scan of the pass's histogram
  uint32_t dbase;
  {
    const uint32_t h = B.ghist[pass * 256 + tid];
    uint32_t incl = h;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += u;
    }
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    dbase = incl - h;
#pragma unroll
    for (int i = 0; i < RADIX_BLOCK / 32; ++i) dbase += i < w ? wsum[i] : 0u;
  }
  uint32_t *st = B.stsort + (size_t)pass * B.nb_radix * 256 + tid;
  for (;;) {
    const uint32_t tile = take_ticket(B.counters + TK_SORT + pass, &slot);
    if (tile >= ntiles) return;
    for (int i = tid; i < (RADIX_BLOCK / 32) * 256; i += RADIX_BLOCK) (&wh[0][0])[i] = 0u;
    __syncthreads();
    uint32_t key[RADIX_ITEMS], val[RADIX_ITEMS];
    int dig[RADIX_ITEMS];
    unsigned peers[RADIX_ITEMS];
    const uint32_t base = tile * RADIX_TILE + w * (32 * RADIX_ITEMS);
#pragma unroll
    for (int r = 0; r < RADIX_ITEMS; ++r) {
      const uint32_t k = base + r * 32 + lane;
      const bool ok = k < V;
      key[r] = ok ? kin[k] : 0u;
      val[r] = ok ? vin[k] : 0u;
    }
#pragma unroll
    for (int r = 0; r < RADIX_ITEMS; ++r) {
      dig[r] = base + r * 32 + lane < V ? (int)((key[r] >> shift) & 255u) : 256;
      peers[r] = digit_peers(dig[r]);
      if (dig[r] < 256 && lane == __ffs(peers[r]) - 1) wh[w][dig[r]] += __popc(peers[r]);
      __syncwarp();
    }
    __syncthreads();
    uint32_t count = 0u;
#pragma unroll
    for (int i = 0; i < RADIX_BLOCK / 32; ++i) count += wh[i][tid];
    st_relaxed(st + (size_t)tile * 256, (tile == 0 ? LB32_INC : LB32_AGG) | count);
    uint32_t excl = 0u;
    bool bad = false;
    if (tile > 0) {
      long long t = (long long)tile - 1;
      bool done = false;
      for (uint32_t polls = 0; !done;) {
        uint32_t word[LB_WIDE];
#pragma unroll
        for (int j = 0; j < LB_WIDE; ++j) word[j] = t - j >= 0 ? ld_relaxed(st + (t - j) * 256) : LB32_INC;
        int adv = 0;
        bool stop = false;
#pragma unroll
        for (int j = 0; j < LB_WIDE; ++j) {
          const uint32_t state = word[j] >> 30;
          stop = stop || state == 0u;
          if (!stop) {
            excl += word[j] & LB32_VAL;
            ++adv;
            done = state == 2u;
            stop = done;
          }
        }
        t -= adv;
        if (!done && adv == 0 && give_up(++polls, B.counters)) {
          bad = true;
          break;
        }
      }
      if (!bad) st_relaxed(st + (size_t)tile * 256, LB32_INC | (excl + count));
    }
    uint32_t run = dbase + excl;
#pragma unroll
    for (int i = 0; i < RADIX_BLOCK / 32; ++i) {
      const uint32_t x = wh[i][tid];
      wh[i][tid] = run;
      run += x;
    }
    if (__syncthreads_or(bad)) {
      if (tid == 0) atomicOr(B.counters + CI_STATUS, ST_GAVE_UP);
      return;
    }
#pragma unroll
    for (int r = 0; r < RADIX_ITEMS; ++r) {
      uint32_t pos = V;
      if (dig[r] < 256) pos = wh[w][dig[r]] + __popc(peers[r] & lanemask_lt());
      __syncwarp();
      if (pos < V) {
        kout[pos] = key[r];
        vout[pos] = val[r];
      }
      if (dig[r] < 256 && lane == __ffs(peers[r]) - 1) wh[w][dig[r]] += __popc(peers[r]);
      __syncwarp();
    }
  }
}

// ---- shared helpers ----------------------------------------------------------

// Inclusive warp prefix sum.
__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(FULL, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Balanced expansion: lane i holds an item with n_i instances (exclusive
// prefix excl_i over the lanes); instance q of the group (item-major order)
// belongs to the largest lane o with excl_o <= q.  Five shuffles.
__device__ __forceinline__ int expansion_owner(int excl, int q) {
  int o = 0;
#pragma unroll
  for (int st = 16; st > 0; st >>= 1) {
    const int e = __shfl_sync(FULL, excl, o + st);
    if (e <= q) o += st;
  }
  return o;
}

// Lanes of `act` whose value v (< 2^nbits) equals this lane's: one ballot
// per bit.
__device__ __forceinline__ unsigned value_peers(int v, int nbits, unsigned act) {
  unsigned m = act;
  for (int b = 0; b < nbits; ++b) {
    const bool bit = (v >> b) & 1;
    const unsigned bb = __ballot_sync(FULL, bit);
    m &= bit ? bb : ~bb;
  }
  return m;
}

__device__ __forceinline__ int bits_for(int n) { return n > 1 ? 32 - __clz(n - 1) : 1; }

// First chunk of row segment sg (of S) when the view has C chunks.
__device__ __forceinline__ uint32_t seg_chunk(int sg, uint32_t C, int S) {
  return (uint32_t)((unsigned long long)sg * C / (unsigned)S);
}

// ---- step 3: equal-work chunks of the depth-sorted list --------------------

// A tile of RADIX_TILE sorted positions per block, eight consecutive ones per
// thread: their packed rectangles are stored in sorted order for every later
// pass, and with p the prefix of the weights (block scan + look-back) and W
// their total (from the compaction), chunk c = the positions whose prefix
// lies in [c W / C, (c + 1) W / C).  Prefixes strictly increase, so the chunk
// of a position never decreases: position s ends the chunks between its own
// and the one its successor's prefix p + weight lies in.  cstart[C] = V.
__global__ void __launch_bounds__(256)
chunk_kernel(const BinViews bv) {
  const BinView &B = bv.v[blockIdx.x];
  const uint32_t V = B.counters[CI_V], ntiles = (V + RADIX_TILE - 1) / RADIX_TILE;
  if (blockIdx.y >= ntiles || stopped(B)) return;
  const uint32_t C = chunk_count(B, V);
  const unsigned long long W = *reinterpret_cast<const unsigned long long *>(B.counters + CI_W);
  __shared__ uint32_t slot;
  __shared__ unsigned long long s_excl;
  __shared__ int s_ok;
  const int tid = threadIdx.x;
  for (;;) {
    const uint32_t tile = take_ticket(B.counters + TK_CHUNK, &slot);
    if (tile >= ntiles) return;
    const uint32_t s0 = tile * RADIX_TILE + tid * CPT;
    uint32_t id[CPT], wt[CPT];
    if (s0 + CPT <= V) {  // s0 % 8 == 0, the array 256-byte aligned
      const uint4 a = *reinterpret_cast<const uint4 *>(B.v0 + s0), b = *reinterpret_cast<const uint4 *>(B.v0 + s0 + 4);
      id[0] = a.x; id[1] = a.y; id[2] = a.z; id[3] = a.w; id[4] = b.x; id[5] = b.y; id[6] = b.z; id[7] = b.w;
    } else {
#pragma unroll
      for (int k = 0; k < CPT; ++k) id[k] = s0 + k < V ? B.v0[s0 + k] : 0u;
    }
    unsigned long long sum = 0;
    uint2 r[CPT];
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      r[k] = make_uint2(0u, 0u);
      if (s0 + k < V) r[k] = reinterpret_cast<const uint2 *>(B.feat + 3 * (size_t)id[k] + 2)[1];
    }
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      wt[k] = s0 + k < V ? chunk_weight(r[k]) : 0u;
      sum += wt[k];
      if (s0 + k < V) B.srect[s0 + k] = r[k];
    }
    unsigned long long total;
    unsigned long long p = block_exclusive_scan<256>(sum, &total);
    if (tid < 32) {
      bool ok;
      const unsigned long long e = lookback(B.stchunk, tile, total, B.counters, &ok);
      if (tid == 0) {
        s_excl = e;
        s_ok = ok;
        if (!ok) atomicOr(B.counters + CI_STATUS, ST_GAVE_UP);
      }
    }
    __syncthreads();
    if (!s_ok) return;
    p += s_excl;
    uint32_t c0 = (uint32_t)(p * C / W);
    if (s0 == 0 && V > 0) {
      B.cstart[0] = 0u;
      B.counters[CI_C] = C;
      if (W > 0xffffffffull) atomicOr(B.counters + CI_STATUS, ST_OVERFLOW);
    }
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
      const uint32_t sp = s0 + k;
      if (sp >= V) break;
      p += wt[k];
      const uint32_t c1 = sp == V - 1 ? C : min((uint32_t)(p * C / W), C);
      for (uint32_t c = c0 + 1; c <= c1; ++c) B.cstart[c] = sp + 1;
      c0 = c1;
    }
  }
}

// ---- steps 4, 5: row counts and segment counts -------------------------------

// Row counts of chunk c, one warp: +1 at the first row and -1 after the last
// of every rectangle in a difference array over the rows, then a prefix sum.
// Written row-major [gy][C] so that one flat exclusive scan gives every
// (row, chunk)'s offset in the concatenated row lists.
__device__ __forceinline__ void row_counts(const BinView &B, uint32_t c, uint32_t C, int *rdiff) {
  const int lane = threadIdx.x & 31, gy = B.gy;
  for (int i = lane; i <= gy; i += 32) rdiff[i] = 0;
  __syncwarp();
  const uint32_t s0 = B.cstart[c], s1 = B.cstart[c + 1];
  for (uint32_t s = s0 + lane; s < s1; s += 32) {
    int x0, y0, x1, y1;
    unpack_rect(B.srect[s], x0, y0, x1, y1);
    if (x0 < x1 && y0 < y1) {
      atomicAdd(&rdiff[y0], 1);
      atomicAdd(&rdiff[y1], -1);
    }
  }
  __syncwarp();
  int carry = 0;
  for (int rb = 0; rb < gy; rb += 32) {
    const int r = rb + lane;
    const int v = warp_incl_scan(r < gy ? rdiff[r] : 0, lane) + carry;
    if (r < gy) B.rcnt[(size_t)r * C + c] = (uint32_t)v;
    carry = __shfl_sync(FULL, v, 31);
  }
}

// Instances of every tile of a band of tile rows from row segment sg (the
// Gaussians of chunks [sg C / S, (sg + 1) C / S)): every rectangle clipped to
// the band adds +1 / -1 at its four corners in a 2D difference grid of
// (R + 1) x (gx + 1) cells (shared-memory atomics from every warp of the
// block); prefix sums along the rows, then the columns, give the counts,
// written to cnt2[t * S + sg] — tile-major, so one flat exclusive scan gives
// every (tile, segment)'s list offset.
__device__ __forceinline__ void segment_counts(const BinView &B, int sg, int b, uint32_t C, int S, int *dg) {
  const int gx = B.gx, ys = b * B.R, ye = min(B.gy, ys + B.R), R = ye - ys, Wd = gx + 1;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int i = tid; i < (R + 1) * Wd; i += 256) dg[i] = 0;
  __syncthreads();
  uint32_t s0 = 0, s1 = 0;
  if (C > 0) {
    s0 = B.cstart[seg_chunk(sg, C, S)];
    s1 = B.cstart[seg_chunk(sg + 1, C, S)];
  }
  for (uint32_t s = s0 + tid; s < s1; s += 256) {
    int x0, y0, x1, y1;
    unpack_rect(B.srect[s], x0, y0, x1, y1);
    const int cy0 = max(y0, ys) - ys, cy1 = min(y1, ye) - ys;
    if (cy0 < cy1 && x0 < x1) {
      atomicAdd(&dg[cy0 * Wd + x0], 1);
      atomicAdd(&dg[cy0 * Wd + x1], -1);
      atomicAdd(&dg[cy1 * Wd + x0], -1);
      atomicAdd(&dg[cy1 * Wd + x1], 1);
    }
  }
  __syncthreads();
  for (int row = w; row < R; row += 8) {  // inclusive prefix along each row
    int carry = 0;
    for (int xb = 0; xb < gx; xb += 32) {
      const int x = xb + lane;
      const int v = warp_incl_scan(x < gx ? dg[row * Wd + x] : 0, lane) + carry;
      if (x < gx) dg[row * Wd + x] = v;
      carry = __shfl_sync(FULL, v, 31);
    }
  }
  __syncthreads();
  for (int x = tid; x < gx; x += 256) {  // inclusive prefix along each column -> counts
    int run = 0;
    for (int row = 0; row < R; ++row) {
      run += dg[row * Wd + x];
      B.cnt2[((size_t)(ys + row) * gx + x) * S + sg] = (uint32_t)run;
    }
  }
}

// Both counts in one launch (each waits on shared memory and on a few loads
// of its own, so they fill one another's gaps): blocks [0, S nb_max) count a
// (segment, band) each, the rest nw chunks' rows each, a warp per chunk.
__global__ void __launch_bounds__(256)
count_kernel(const BinViews bv, int S, int nb_max, int nw) {
  extern __shared__ int cnt_smem[];
  const BinView &B = bv.v[blockIdx.y];
  if (B.counters[CI_STATUS] & ST_STOP) return;  // block-uniform: no block of this launch sets a bit
  const uint32_t C = chunk_count(B, B.counters[CI_V]);
  if ((int)blockIdx.x < S * nb_max) {
    if ((int)blockIdx.x < S * B.nb)  // block-uniform
      segment_counts(B, (int)blockIdx.x / B.nb, (int)blockIdx.x % B.nb, C, S, cnt_smem);
    return;
  }
  const int w = threadIdx.x >> 5;
  const uint32_t c = (blockIdx.x - S * nb_max) * nw + w;
  if (w < nw && c < C) row_counts(B, c, C, cnt_smem + w * (B.gy + 1));
}

// Exclusive scans in place of the row counts [gy][C] (total: the row-list
// entries K1) and of the segment counts [T][S] (total: the instances K), in
// tiles of SCAN_TILE: the row counts' tiles first, then the segment counts',
// each array with its own chain of look-back words.
__global__ void __launch_bounds__(SCAN_THREADS)
list_scan_kernel(const BinViews bv, int S) {
  const BinView &B = bv.v[blockIdx.x];
  if (stopped(B)) return;
  const uint32_t C = chunk_count(B, B.counters[CI_V]);
  const size_t nr = (size_t)B.gy * C, ns = (size_t)B.gx * B.gy * S;
  const uint32_t tr = (uint32_t)scan_tiles(nr), ts = (uint32_t)scan_tiles(ns);
  __shared__ uint32_t slot;
  __shared__ unsigned long long s_excl;
  __shared__ int s_ok;
  const int tid = threadIdx.x;
  if (blockIdx.y >= tr + ts) return;  // block-uniform
  for (;;) {
    const uint32_t tile = take_ticket(B.counters + TK_SCAN, &slot);
    if (tile >= tr + ts) return;
    const bool rows = tile < tr;
    uint32_t *data = rows ? B.rcnt : B.cnt2;
    const size_t n = rows ? nr : ns;
    const uint32_t t = rows ? tile : tile - tr;
    unsigned long long *st = B.stscan + (rows ? 0 : scan_tiles((size_t)B.gy * CHUNK_COUNT_MAX));
    const size_t k0 = (size_t)t * SCAN_TILE + tid * SCAN_ITEMS;
    static_assert(SCAN_ITEMS == 4, "a thread's items are one 16-byte word");
    uint4 x = make_uint4(0u, 0u, 0u, 0u);
    const bool whole = k0 + 4 <= n;  // k0 % 4 == 0, the arrays 256-byte aligned
    if (whole) {
      x = *reinterpret_cast<const uint4 *>(data + k0);
    } else {
      if (k0 < n) x.x = data[k0];
      if (k0 + 1 < n) x.y = data[k0 + 1];
      if (k0 + 2 < n) x.z = data[k0 + 2];
    }
    unsigned long long total;
    unsigned long long run = block_exclusive_scan<SCAN_THREADS>(
        (unsigned long long)x.x + x.y + x.z + x.w, &total);
    if (tid < 32) {
      bool ok;
      const unsigned long long e = lookback(st, t, total, B.counters, &ok);
      if (tid == 0) {
        s_excl = e;
        s_ok = ok;
        if (!ok) atomicOr(B.counters + CI_STATUS, ST_GAVE_UP);
        if (ok && t == (rows ? tr : ts) - 1) {
          B.counters[rows ? CI_K1 : CI_K] = (uint32_t)(e + total);
          if (e + total > 0xffffffffull) atomicOr(B.counters + CI_STATUS, ST_OVERFLOW);
        }
      }
    }
    __syncthreads();
    if (!s_ok) return;
    const uint32_t r0 = (uint32_t)(run + s_excl), r1 = r0 + x.x, r2 = r1 + x.y, r3 = r2 + x.z;
    if (whole) {
      *reinterpret_cast<uint4 *>(data + k0) = make_uint4(r0, r1, r2, r3);
    } else {
      if (k0 < n) data[k0] = r0;
      if (k0 + 1 < n) data[k0 + 1] = r1;
      if (k0 + 2 < n) data[k0 + 2] = r2;
    }
  }
}

// Tile ranges from the scanned segment counts: tile t starts at its first
// segment's offset.  When the instances exceed the list capacity
// (capacity-bounded callers), every range is left empty and the overflow bit
// is set, so no kernel reads past the list buffer.
__global__ void ranges_kernel(const BinViews bv, int S) {
  const BinView &B = bv.v[blockIdx.y];
  const int T = B.gx * B.gy;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  uint32_t *counters = B.counters;
  const uint32_t K = counters[CI_K];
  const uint32_t status = counters[CI_STATUS];
  const bool over = K > B.K_cap || (status & ST_STOP);
  if (t == 0 && (K > B.K_cap || (status & ST_OVERFLOW))) atomicOr(&counters[CI_STATUS], ST_OVERFLOW);
  uint2 r = make_uint2(0u, 0u);
  if (B.P > 0 && !over) {
    const uint32_t a = B.cnt2[(size_t)t * S];
    const uint32_t e = (t + 1 < T) ? B.cnt2[(size_t)(t + 1) * S] : K;
    if (e > a) r = make_uint2(a, e);
    atomicMax(&counters[CI_MAXLIST], e - a);
  }
  B.ranges[t] = r;
  // the tile's class, by half octaves of its length
  int c = BLEND_CLASSES - 1;
  if (r.y > r.x) {
    const uint32_t n = r.y - r.x;
    const int l = 31 - __clz(n), b = 2 * l + (l > 0 ? (int)((n >> (l - 1)) & 1u) : 0);
    c = max(0, BLEND_CLASSES - 2 - b);
  }
  B.clslist[class_slot(c, atomicAdd(&B.clsn[c], 1u), T)] = (uint32_t)t;
}

// ---- step 6a: row lists, one warp per chunk --------------------------------

// The chunk's Gaussians are taken 32 at a time (depth order); the (Gaussian,
// row) pairs of the group are spread over the lanes in Gaussian-major order
// (balanced expansion), so pairs of one row rank by their Gaussian's depth
// order: rank = lanes of lower index in the same row (a ballot per bit), then the row's
// running slot (shared memory) advances by the row's pairs.
__global__ void __launch_bounds__(32)
row_emit_kernel(const BinViews bv) {
  extern __shared__ uint32_t rcur[];  // gy running slots
  const BinView &B = bv.v[blockIdx.y];
  uint32_t *counters = B.counters;
  const uint32_t C = counters[CI_C];
  const uint32_t c = blockIdx.x;
  if (c >= C || __any_sync(FULL, (counters[CI_STATUS] & ST_STOP) != 0u)) return;  // one warp a block
  const int lane = threadIdx.x, gy = B.gy, nbits = bits_for(gy);
  for (int r = lane; r < gy; r += 32) rcur[r] = B.rcnt[(size_t)r * C + c];
  __syncwarp();
  const uint32_t s0 = B.cstart[c], s1 = B.cstart[c + 1];
  const uint32_t cap = B.rows_alloc;
  const uint2 *__restrict__ srect = B.srect;
  const uint32_t *__restrict__ order = B.v0;
  uint2 *__restrict__ rowlist = B.rowlist;
  const unsigned lt = lanemask_lt();
  bool bad = false;
  for (uint32_t g0 = s0; g0 < s1; g0 += 32) {
    const uint32_t s = g0 + lane;
    const bool v = s < s1;
    const uint2 rr = v ? srect[s] : make_uint2(0u, 0u);
    const uint32_t id = v ? order[s] : 0u;
    int x0, y0, x1, y1;
    unpack_rect(rr, x0, y0, x1, y1);
    const int n = (x0 < x1 && y0 < y1) ? y1 - y0 : 0;
    const int incl = warp_incl_scan(n, lane);
    const int total = __shfl_sync(FULL, incl, 31);
    const int excl = incl - n;
    const uint32_t xr = (rr.x & 0xffffu) | (rr.y << 16);
    for (int base = 0; base < total; base += 32) {
      const int q = base + lane;
      const bool act = q < total;
      const int o = expansion_owner(excl, q);
      const int row = __shfl_sync(FULL, y0, o) + (q - __shfl_sync(FULL, excl, o));
      const uint32_t ido = __shfl_sync(FULL, id, o);
      const uint32_t xro = __shfl_sync(FULL, xr, o);
      const unsigned amask = total - base >= 32 ? FULL : (1u << (total - base)) - 1u;
      const unsigned peers = value_peers(act ? row : 0, nbits, amask);
      const uint32_t p = act ? rcur[row] + __popc(peers & lt) : 0u;
      __syncwarp();
      if (act) {
        if (p < cap) rowlist[p] = make_uint2(ido, xro); else bad = true;
        if ((peers & lt) == 0u) rcur[row] += __popc(peers);
      }
      __syncwarp();
    }
  }
  if (bad) atomicOr(&counters[CI_STATUS], ST_BOUNDS);
}

// ---- step 6b: tile lists, one block per (tile row, row piece, segment) -----

constexpr int TE_WARPS = 8;
constexpr int TE_THREADS = 32 * TE_WARPS;
constexpr int STAGE_CAP = 8192;    // staged instances per sub-pass
constexpr int TE_COPY = 8;         // lanes copying a tile's staged run
constexpr int TE_PER = 4;          // row-list entries per thread considered for a sub-pass
constexpr int TE_ENTRIES = TE_THREADS * TE_PER;

__host__ __device__ inline size_t tile_emit_smem_words(int nx) {
  return (size_t)nx + (nx + 1) + (size_t)TE_WARPS * (nx + 1) + STAGE_CAP + TE_WARPS +
         (TE_WARPS + 1) + (size_t)TE_WARPS * ((size_t)nx + 32);
}

__device__ __forceinline__ int block_sum_te(int v, int *red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  int t = 0;
#pragma unroll
  for (int i = 0; i < TE_WARPS; ++i) t += red[i];
  return t;
}

// The block's entries (one segment of one row list, depth order) are split
// into sub-passes whose instances fit the staging buffer; per sub-pass, each
// warp takes a contiguous slice of entries (about equal instance counts):
// (A) per-warp counts per tile (1D difference array); (B) per tile the
// exclusive prefix over the warps and the tiles' staging offsets, giving
// every warp an absolute staging cursor per tile; (C) the slice's entries in
// order, one at a time, each writing its Gaussian index at the cursor of
// every tile it covers (tile x always by lane x % 32, so no two lanes share
// a cursor and no ranks are needed); (D) each tile's staged run copied to
// the tile's list at its running position (coalesced).
// Bound by issue (73% of the slots): the block's fixed work and the XOR scans.
// 16 views of 3M Gaussians (176M instances): 707 us with a scan each for the
// begun and the ended entries, 64-bit slice cuts and a warp per copied run,
// 608 us so; four views of 500k 82 -> 53 us, one of 3M 74 -> 66 us.
__global__ void __launch_bounds__(TE_THREADS)
tile_emit_kernel(const BinViews bv, int S) {
  extern __shared__ uint32_t te[];
  const BinView &B = bv.v[blockIdx.y];
  const int sg = blockIdx.x % S, rest = blockIdx.x / S;
  const int xs = rest % B.nxs, r = rest / B.nxs;
  if (r >= B.gy) return;  // block-uniform
  uint32_t *counters = B.counters;
  const uint32_t C = counters[CI_C];
  if (C == 0 || stopped(B)) return;
  const uint32_t f0 = seg_chunk(sg, C, S), f1 = seg_chunk(sg + 1, C, S);
  if (f0 >= f1) return;
  const uint32_t e0 = B.rcnt[(size_t)r * C + f0];
  const uint32_t e1 = f1 < C ? B.rcnt[(size_t)r * C + f1]
                             : (r + 1 < B.gy ? B.rcnt[(size_t)(r + 1) * C] : counters[CI_K1]);
  if (e0 >= e1) return;
  const int xa = xs * XSEG, nx = min(B.gx - xa, XSEG);
  uint32_t *tcur = te;                                   // [nx] running list positions
  uint32_t *soff = tcur + nx;                            // [nx + 1] staging offsets
  int *wc = reinterpret_cast<int *>(soff + nx + 1);      // [TE_WARPS][nx + 1] counts / cursors
  uint32_t *stage = reinterpret_cast<uint32_t *>(wc + TE_WARPS * (nx + 1));  // [STAGE_CAP]
  int *red = reinterpret_cast<int *>(stage + STAGE_CAP);  // [TE_WARPS]
  uint32_t *bnd = reinterpret_cast<uint32_t *>(red + TE_WARPS);  // [TE_WARPS + 1] slice starts
  // per warp: the entries whose cover changes at a tile [nx] (zero between
  // groups) and the Gaussian indices of the current group of 32 entries
  uint32_t *smask = bnd + TE_WARPS + 1;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  uint32_t *tog = smask + (size_t)w * (nx + 32), *gids = tog + nx;
  for (int i = tid; i < TE_WARPS * (nx + 32); i += TE_THREADS) smask[i] = 0u;
  const uint2 *__restrict__ rl = B.rowlist;
  uint32_t *__restrict__ out = B.point_list;
  const uint32_t cap = B.K_alloc;
  for (int x = tid; x < nx; x += TE_THREADS)
    tcur[x] = B.cnt2[((size_t)r * B.gx + xa + x) * S + sg];
  int *wcw = wc + w * (nx + 1);
  bool bad = false;
  auto clip = [&](uint2 en, int &a, int &b) {
    a = max((int)(en.y & 0xffffu), xa) - xa;
    b = min((int)(en.y >> 16), xa + nx) - xa;
  };
  for (uint32_t e = e0; e < e1;) {
    // sub-pass: the longest run of entries whose instances fit the staging
    // buffer (block scan of the clipped widths of up to TE_ENTRIES entries),
    // cut into one contiguous slice per warp at equal instance counts
    const uint32_t navail = min(e1 - e, (uint32_t)TE_ENTRIES);
    int wd[TE_PER];
    int tsum = 0;
#pragma unroll
    for (int k = 0; k < TE_PER; ++k) {
      const uint32_t i = (uint32_t)tid * TE_PER + k;
      int a = 0, b = 0;
      if (i < navail) clip(rl[e + i], a, b);
      wd[k] = max(b - a, 0);
      tsum += wd[k];
    }
    const int tin = warp_incl_scan(tsum, lane);
    __syncthreads();  // red[] and bnd[] of the previous sub-pass are no longer read
    if (lane == 31) red[w] = tin;
    if (tid <= TE_WARPS) bnd[tid] = 0xffffffffu;
    __syncthreads();
    int wbase = 0, itot = 0;
#pragma unroll
    for (int i = 0; i < TE_WARPS; ++i) {
      wbase += i < w ? red[i] : 0;
      itot += red[i];
    }
    int run = wbase + tin - tsum;  // instances before this thread's entries
    int fit = 0;
#pragma unroll
    for (int k = 0; k < TE_PER; ++k) {
      run += wd[k];
      fit += (run <= STAGE_CAP && (uint32_t)tid * TE_PER + k < navail) ? 1 : 0;
    }
    const uint32_t En = max(1u, (uint32_t)block_sum_te(fit, red));
    const int I = min(itot, STAGE_CAP);  // instances of the first En entries (all of them when they fit)
    {
      int ex = wbase + tin - tsum;
#pragma unroll
      for (int k = 0; k < TE_PER; ++k) {
        const uint32_t i = (uint32_t)tid * TE_PER + k;
        if (i < En && I > 0) {
          // ex <= STAGE_CAP here: the product stays below 2^32
          const int wi = (int)((uint32_t)ex * TE_WARPS / (uint32_t)I);
          atomicMin(&bnd[min(wi, TE_WARPS - 1)], i);
        }
        ex += wd[k];
      }
    }
    __syncthreads();
    // slice starts: first entry whose instances begin in the warp's share
    // (a slice without one starts where the next does)
    uint32_t bm = lane > 0 && lane < TE_WARPS ? bnd[lane] : (lane == 0 ? 0u : En);
#pragma unroll
    for (int o = 1; o < TE_WARPS; o <<= 1) bm = min(bm, __shfl_down_sync(FULL, bm, o));
    const uint32_t sa = e + __shfl_sync(FULL, bm, w), sb = e + __shfl_sync(FULL, bm, w + 1);
    // (A) this warp's counts per tile
    for (int i = lane; i <= nx; i += 32) wcw[i] = 0;
    __syncwarp();
    for (uint32_t i = sa + lane; i < sb; i += 32) {
      int a, b;
      clip(rl[i], a, b);
      if (a < b) {
        atomicAdd(&wcw[a], 1);
        atomicAdd(&wcw[b], -1);
      }
    }
    __syncwarp();
    {
      int carry = 0;
      for (int xb = 0; xb < nx; xb += 32) {
        const int x = xb + lane;
        const int v = warp_incl_scan(x < nx ? wcw[x] : 0, lane) + carry;
        if (x < nx) wcw[x] = v;
        carry = __shfl_sync(FULL, v, 31);
      }
    }
    __syncthreads();
    // (B) per tile: prefix over the warps, tile totals, staging offsets
    for (int x = tid; x < nx; x += TE_THREADS) {
      int run = 0;
#pragma unroll
      for (int w2 = 0; w2 < TE_WARPS; ++w2) {
        const int cw = wc[w2 * (nx + 1) + x];
        wc[w2 * (nx + 1) + x] = run;
        run += cw;
      }
      soff[x] = (uint32_t)run;
    }
    __syncthreads();
    if (w == 0) {  // exclusive scan of the tile totals (nx <= XSEG)
      uint32_t carry = 0;
      for (int xb = 0; xb < nx; xb += 32) {
        const int x = xb + lane;
        const int t = x < nx ? (int)soff[x] : 0;
        const int incl = warp_incl_scan(t, lane);
        if (x < nx) soff[x] = carry + (uint32_t)(incl - t);
        carry += (uint32_t)__shfl_sync(FULL, incl, 31);
      }
      if (lane == 0) soff[nx] = carry;
    }
    __syncthreads();
    for (int x = lane; x < nx; x += 32) wcw[x] += (int)soff[x];  // the warp's absolute staging cursors
    __syncwarp();
    // (C) stage the slice's instances, 32 entries (depth order) at a time:
    // lane j flips bit j at its entry's first tile a_j and at its end b_j;
    // the inclusive XOR-prefix over the tiles is the set of entries that
    // cover a tile, which the lane owning tile x (x % 32) appends in bit
    // (entry) order at its cursor — so a tile's cursor is only ever touched
    // by one lane and entries land in the order they come.
    for (uint32_t g0 = sa; g0 < sb; g0 += 32) {
      const uint32_t i = g0 + lane;
      const uint2 en = i < sb ? rl[i] : make_uint2(0u, 0u);
      int a = 0, b = 0;
      if (i < sb) clip(en, a, b);
      const bool has = a < b;
      gids[lane] = en.x;
      if (has) {
        atomicXor(&tog[a], 1u << lane);
        if (b < nx) atomicXor(&tog[b], 1u << lane);  // an end at nx is never read
      }
      const int lo = (int)__reduce_min_sync(FULL, has ? (unsigned)a : 0xffffffffu);
      const int hi = (int)__reduce_max_sync(FULL, has ? (unsigned)b : 0u);
      __syncwarp();
      // none of the group's entries may lie in this piece of a row of more than
      // XSEG tiles: hi is 0 then, and lo no tile
      if (hi > 0) {  // warp-uniform; chunks up to the one holding hi (clears tog[hi])
        uint32_t carry = 0u;
        for (int xb = lo & ~31; xb <= hi && xb < nx; xb += 32) {
          const int x = xb + lane;
          uint32_t mm = x < nx ? tog[x] : 0u;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(FULL, mm, o);
            if (lane >= o) mm ^= u;
          }
          mm ^= carry;
          carry = __shfl_sync(FULL, mm, 31);
          if (x < nx) {
            tog[x] = 0u;
            if (mm) {
              uint32_t p = (uint32_t)wcw[x];
              do {
                const int j = __ffs(mm) - 1;
                mm &= mm - 1;
                if (p < STAGE_CAP) stage[p] = gids[j]; else bad = true;
                ++p;
              } while (mm);
              wcw[x] = (int)p;
            }
          }
        }
      }
      __syncwarp();
    }
    __syncthreads();
    // (D) copy each tile's staged run to its list, TE_COPY lanes a tile
    // (runs are some ten to a hundred instances long)
    for (int x = w * (32 / TE_COPY) + lane / TE_COPY; x < nx; x += TE_WARPS * (32 / TE_COPY)) {
      const uint32_t a = soff[x], n = soff[x + 1] - a, dst = tcur[x];
      for (uint32_t j = lane % TE_COPY; j < n; j += TE_COPY) {
        if (dst + j < cap) out[dst + j] = stage[a + j]; else bad = true;
      }
    }
    __syncthreads();
    for (int x = tid; x < nx; x += TE_THREADS) tcur[x] += soff[x + 1] - soff[x];
    e += En;
  }
  if (bad) atomicOr(&counters[CI_STATUS], ST_BOUNDS);
}

// Debug view: sorted keys in the reference's form (tile << 32 | depth_bits).
__global__ void debug_keys_kernel(int T, const uint2 *__restrict__ ranges,
                                  const uint32_t *__restrict__ point_list,
                                  const float4 *__restrict__ feat, uint64_t *__restrict__ keys_out,
                                  uint32_t *__restrict__ values_out) {
  const int t = blockIdx.x;
  const uint2 r = ranges[t];
  for (uint32_t i = r.x + threadIdx.x; i < r.y; i += blockDim.x) {
    const uint32_t id = point_list[i];
    if (keys_out) keys_out[i] = ((uint64_t)t << 32) | __float_as_uint(feat[3 * id + 2].y);
    if (values_out) values_out[i] = id;
  }
}


}  // namespace

namespace {

// Bands of tile rows for the segment counts: about 1024 tiles per band (a
// 4 KB difference grid).
void band_plan(int gx, int gy, int &R, int &nb) {
  R = std::max(1, std::min(gy, 1024 / std::max(gx, 1)));
  nb = (gy + R - 1) / R;
}

size_t seg_grid_bytes(int R, int gx) { return (size_t)(R + 1) * (gx + 1) * 4; }

int device_sms() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return NUM_SMS_HINT;
  thread_local int cached_dev = -1, cached_sms = NUM_SMS_HINT;
  if (dev != cached_dev) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0)
      cached_sms = sms;
    cached_dev = dev;
  }
  return cached_sms;
}

// Row segments per view for a launch: enough (row, piece, segment) blocks for
// several waves of the tile emission (short blocks balance uneven rows), but
// not so many that a block's fixed work (sub-pass cut, cursors, run copies)
// outweighs its instances.  Where the two meet moves with the work: the best
// count grows about as the root of the Gaussians x views.  Counts, scans and
// emission together, us, at 16 | 24 | 32 | 48 blocks an SM and (this rule's):
//   4 views of 0.25M, 0.5M, 1M, 2M   73 | 81 | 90 | 111 (16), 96 | 97 | 105 | 124 (16), 146 | 136 | 138 | 153 (22), 253 | 228 | 220 | 229 (31)
//   8 views of the same              92 | 95 | 105 | 125 (16), 140 | 135 | 136 | 150 (22), 229 | 208 | 200 | 206 (31), 410 | 363 | 342 | 334 (44)
//   16 views of the same             120 | 123 | 126 | 147 (22), 193 | 182 | 182 | 196 (31), 347 | 315 | 311 | 313 (44), 637 | 579 | 560 | 545 (48)
// at 1237 x 822, and at 400 x 300, 200 x 200 and 3000 x 2000 with 0.1M and 1M
// the same order.  A single view is at SEG_MAX on most grids.  A pure function
// of the views' grids and sizes and the device, so the geometry and the
// emission launches of one set of views agree.
int seg_plan(const BinViews &bv) {
  long rows = 0, gaussians = 0;
  for (int v = 0; v < bv.n; ++v) {
    rows += (long)bv.v[v].gy * bv.v[v].nxs;
    gaussians += bv.v[v].P;
  }
  const double per_sm = std::min(48.0, std::max(16.0, 16.0 * std::sqrt((double)gaussians / (double)(1 << 21))));
  const long target = (long)per_sm * device_sms();
  const long S = rows > 0 ? (target + rows - 1) / rows : 1;
  return (int)std::max(1L, std::min((long)SEG_MAX, S));
}

// Blocks per view for a grid-stride launch over at most `units` work units
// whose actual count is only known on the device: about two resident waves
// of `per_sm` blocks per SM shared by the views, so that a launch sized for
// the worst case does not schedule thousands of blocks that find no work.
int bounded_blocks(size_t units, int nviews, int per_sm) {
  const size_t cap = std::max<size_t>(1, (size_t)2 * device_sms() * per_sm / std::max(nviews, 1));
  return (int)std::max<size_t>(1, std::min(units, cap));
}

constexpr size_t SMEM_LIMIT = 220 * 1024;

}  // namespace

int launch_scan1(uint32_t *data, uint32_t n, uint32_t *part, uint32_t *total_out, cudaStream_t s) {
  if (n <= (uint32_t)SCAN_TILE * 4) {
    dmgs_host::note_launch(), scan_single_kernel<<<1, SCAN_THREADS, 0, s>>>(data, n, total_out);
    DMGS_LAUNCH_CHECK("scan_single_kernel");
    return DMGS_OK;
  }
  const uint32_t tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  const int grid = bounded_blocks(tiles, 1, 2);
  dmgs_host::note_launch(), scan_reduce_kernel<<<grid, SCAN_THREADS, 0, s>>>(data, n, part);
  DMGS_LAUNCH_CHECK("scan_reduce_kernel");
  dmgs_host::note_launch(), scan_single_kernel<<<1, SCAN_THREADS, 0, s>>>(part, tiles, total_out);
  DMGS_LAUNCH_CHECK("scan_single_kernel");
  dmgs_host::note_launch(), scan_down_kernel<<<grid, SCAN_THREADS, 0, s>>>(data, n, part);
  DMGS_LAUNCH_CHECK("scan_down_kernel");
  return DMGS_OK;
}

size_t scan_part_words(uint32_t n) { return (n + SCAN_TILE - 1) / SCAN_TILE + 1; }

int make_bin_view(const GeomLayout &L, char *geom, uint32_t K_cap, char *bin, uint32_t K_alloc,
                  BinView &B) {
  B.P = L.P;
  B.nb_radix = L.nb_radix;
  B.gx = L.gx;
  B.gy = L.gy;
  band_plan(L.gx, L.gy, B.R, B.nb);
  B.nxs = (L.gx + XSEG - 1) / XSEG;
  const size_t rows_smem = (size_t)(L.gy + 1) * 4;
  if (seg_grid_bytes(B.R, L.gx) > SMEM_LIMIT || rows_smem > SMEM_LIMIT) {
    dmgs_host::set_error("image too large for the binning kernels' shared memory (%d x %d tiles)",
                         L.gx, L.gy);
    return DMGS_ERR_ARG;
  }
  B.flags = reinterpret_cast<const uint8_t *>(geom + L.flags);
  B.feat = reinterpret_cast<const float4 *>(geom + L.feat);
  B.counters = reinterpret_cast<uint32_t *>(geom + L.counters);
  B.ghist = reinterpret_cast<uint32_t *>(geom + L.ghist);
  B.stsort = reinterpret_cast<uint32_t *>(geom + L.stsort);
  B.clsn = reinterpret_cast<uint32_t *>(geom + L.clsn);
  B.clslist = reinterpret_cast<uint32_t *>(geom + L.clslist);
  B.vtile = reinterpret_cast<uint32_t *>(geom + L.vtile);
  B.vgroup = reinterpret_cast<uint32_t *>(geom + L.vgroup);
  B.stchunk = reinterpret_cast<unsigned long long *>(geom + L.stchunk);
  B.stscan = reinterpret_cast<unsigned long long *>(geom + L.stscan);
  B.vlist = reinterpret_cast<uint32_t *>(geom + L.vlist);
  B.k0 = reinterpret_cast<uint32_t *>(geom + L.dkey0);
  B.k1 = reinterpret_cast<uint32_t *>(geom + L.dkey1);
  B.v0 = reinterpret_cast<uint32_t *>(geom + L.dval0);
  B.v1 = reinterpret_cast<uint32_t *>(geom + L.dval1);
  B.srect = reinterpret_cast<uint2 *>(geom + L.srect);
  B.cstart = reinterpret_cast<uint32_t *>(geom + L.cstart);
  B.rcnt = reinterpret_cast<uint32_t *>(geom + L.rcnt);
  B.cnt2 = reinterpret_cast<uint32_t *>(geom + L.cnt2);
  B.ranges = reinterpret_cast<uint2 *>(geom + L.ranges);
  // the caller sized the state with bin_layout(K_alloc, ...) (plain form: K
  // row entries) or bin_layout(K_alloc, ..., P) (capacity-bounded forms:
  // fewer); the smaller bound is always inside the buffer
  const BinLayout BL = bin_layout(K_alloc, L.gx * TILE, L.gy * TILE, L.P);
  B.point_list = bin ? reinterpret_cast<uint32_t *>(bin + BL.point_list) : nullptr;
  B.rowlist = bin ? reinterpret_cast<uint2 *>(bin + BL.rowlist) : nullptr;
  B.K_cap = K_cap;
  B.K_alloc = bin ? K_alloc : 0u;
  B.rows_alloc = bin ? (uint32_t)BL.rows : 0u;
  B.cmax = CHUNK_COUNT_MAX;
  return DMGS_OK;
}

int launch_binning_geometry(const BinViews &bv, cudaStream_t s) {
  if (bv.n < 1) return DMGS_OK;
  int nb_radix = 0, P = 0, T = 0, gy = 0, nb = 0;
  uint32_t cmax = 0;
  size_t seg_smem = 0;
  for (int v = 0; v < bv.n; ++v) {
    const BinView &B = bv.v[v];
    nb_radix = std::max(nb_radix, B.nb_radix);
    P = std::max(P, B.P);
    T = std::max(T, B.gx * B.gy);
    gy = std::max(gy, B.gy);
    nb = std::max(nb, B.nb);
    cmax = std::max(cmax, B.cmax);
    seg_smem = std::max(seg_smem, seg_grid_bytes(B.R, B.gx));
  }
  const int S = seg_plan(bv);
  const int nv = bv.n;
  if (P > 0) {
    // tiles of the visible Gaussians, whose number is known on the device
    const int tgrid = bounded_blocks((size_t)nb_radix, nv, 8);
    // chunk warps of a counting block: as many rows as 48 KB hold, 1 to 8
    const size_t row_smem = (size_t)(gy + 1) * 4;
    const int nw = (int)std::max<size_t>(1, std::min<size_t>(8, 48 * 1024 / row_smem));
    const size_t cnt_smem = std::max(seg_smem, nw * row_smem);
    if (int r = dmgs_host::raise_smem_limit((const void *)count_kernel, cnt_smem)) return r;
    const size_t st_max = scan_tiles((size_t)gy * cmax) + scan_tiles((size_t)T * S);
    DMGS_TIMED(K_BIN_COMPACT, s,
               dmgs_host::note_launch(), compact_kernel<<<dim3(nv, std::min(nb_radix, 65535)), PRE_BLOCK, 0, s>>>(bv));
    DMGS_LAUNCH_CHECK("compact_kernel");
    DMGS_TIMED(K_BIN_SORT, s, {
      for (int pass = 0; pass < 4; ++pass)
        dmgs_host::note_launch(), radix_pass_kernel<<<dim3(nv, tgrid), RADIX_BLOCK, 0, s>>>(bv, pass);
    });  // four passes: the sorted order ends in (k0, v0)
    DMGS_LAUNCH_CHECK("radix_sort");
    DMGS_TIMED(K_BIN_COUNT, s, {
      dmgs_host::note_launch(), chunk_kernel<<<dim3(nv, tgrid), 256, 0, s>>>(bv);
      dmgs_host::note_launch(), count_kernel<<<dim3(S * nb + (cmax + nw - 1) / nw, nv), 256, cnt_smem, s>>>(bv, S, nb, nw);
    });
    DMGS_LAUNCH_CHECK("tile_count");
    DMGS_TIMED(K_BIN_SCAN, s,
               dmgs_host::note_launch(), list_scan_kernel<<<dim3(nv, bounded_blocks(st_max, nv, 2)), SCAN_THREADS, 0, s>>>(bv, S));
    DMGS_LAUNCH_CHECK("binning scans");
  }
  dmgs_host::note_launch(), ranges_kernel<<<dim3((T + 255) / 256, nv), 256, 0, s>>>(bv, S);
  DMGS_LAUNCH_CHECK("ranges_kernel");
  return DMGS_OK;
}

int launch_emit(const BinViews &bv, cudaStream_t s) {
  int gy = 0, nxs = 0, gxm = 0;
  uint32_t cmax = 0;
  bool any = false;
  for (int v = 0; v < bv.n; ++v) {
    const BinView &B = bv.v[v];
    if (B.P <= 0 || B.K_alloc == 0) continue;
    any = true;
    gy = std::max(gy, B.gy);
    nxs = std::max(nxs, B.nxs);
    gxm = std::max(gxm, std::min(B.gx, XSEG));
    cmax = std::max(cmax, B.cmax);
  }
  if (!any) return DMGS_OK;
  const int S = seg_plan(bv);
  const size_t rows_smem = (size_t)gy * 4;
  const size_t te_smem = tile_emit_smem_words(gxm) * 4;
  if (int r = dmgs_host::raise_smem_limit((const void *)row_emit_kernel, rows_smem)) return r;
  if (int r = dmgs_host::raise_smem_limit((const void *)tile_emit_kernel, te_smem)) return r;
  DMGS_TIMED(K_BIN_ROWS, s,
             dmgs_host::note_launch(), row_emit_kernel<<<dim3(cmax, bv.n), 32, rows_smem, s>>>(bv));
  DMGS_LAUNCH_CHECK("row_emit_kernel");
  DMGS_TIMED(K_BIN_EMIT, s,
             dmgs_host::note_launch(), tile_emit_kernel<<<dim3(gy * nxs * S, bv.n), TE_THREADS, te_smem, s>>>(bv, S));
  DMGS_LAUNCH_CHECK("tile_emit_kernel");
  return DMGS_OK;
}

int launch_debug_keys(const GeomLayout &L, const char *geom, const BinLayout &B, const char *bin,
                      uint64_t *keys, uint32_t *values, cudaStream_t s) {
  DMGS_TIMED(K_DEBUG, s, dmgs_host::note_launch(), debug_keys_kernel<<<L.T(), 256, 0, s>>>(
      L.T(), reinterpret_cast<const uint2 *>(geom + L.ranges),
      reinterpret_cast<const uint32_t *>(bin + B.point_list),
      reinterpret_cast<const float4 *>(geom + L.feat), keys, values));
  DMGS_LAUNCH_CHECK("debug_keys_kernel");
  return DMGS_OK;
}

}  // namespace dmgs
