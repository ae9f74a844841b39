// The binning's look-back kernels on a state whose first tile is never taken:
// its ticket counter starts at 1, so every later tile waits for a word that no
// block publishes, until its polls run out.  Built by the test with a lower
// limit (DMGS_LB_POLLS); every access is in bounds (the state has the layout
// and size of a view's), and the waits end by the limit.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../dmgs_gb300/csrc/binning.cu"

namespace dmgs_host {
void set_error(const char *, ...) {}
int cuda_fail(cudaError_t e, const char *what) { fprintf(stderr, "%s: %s\n", what, cudaGetErrorString(e)); return DMGS_ERR_CUDA; }
void timing_begin(int, cudaStream_t) {}
void timing_end(int, cudaStream_t) {}
void note_launch() {}
int raise_smem_limit(const void *f, size_t bytes) {
  return bytes > 48 * 1024 ? (int)cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) : 0;
}
}  // namespace dmgs_host

using namespace dmgs;

#define OK(x) do { cudaError_t e_ = (x); if (e_ != cudaSuccess) { fprintf(stderr, "%s: %s\n", #x, cudaGetErrorString(e_)); exit(2); } } while (0)

struct State {
  GeomLayout L;
  char *geom;
  BinViews bv;
  uint32_t *word(size_t off, int i) { return reinterpret_cast<uint32_t *>(geom + off) + i; }
  void set(size_t off, int i, uint32_t v) { OK(cudaMemcpy(word(off, i), &v, 4, cudaMemcpyHostToDevice)); }
  uint32_t get(size_t off, int i) { uint32_t v; OK(cudaMemcpy(&v, word(off, i), 4, cudaMemcpyDeviceToHost)); return v; }
};

// All P Gaussians visible, the list 0, 1, 2, ... in place, records of zeros.
static State make(int P, int W, int H) {
  State s;
  s.L = geom_layout(P, W, H);
  OK(cudaMalloc(&s.geom, s.L.total));
  OK(cudaMemset(s.geom, 0, s.L.total));
  std::vector<uint32_t> ids(P);
  for (int i = 0; i < P; ++i) ids[i] = i;
  OK(cudaMemcpy(s.geom + s.L.dval0, ids.data(), 4 * (size_t)P, cudaMemcpyHostToDevice));
  s.set(s.L.counters, CI_V, P);
  s.set(s.L.counters, CI_W, 2 * P);
  s.bv.n = 1;
  if (make_bin_view(s.L, s.geom, 0xffffffffu, nullptr, 0u, s.bv.v[0])) exit(2);
  return s;
}

int main() {
  const int P = 5 * RADIX_TILE - 7, W = 640, H = 480;
  int rc = 0;
  for (int which = 0; which < 4; ++which) {
    State s = make(P, W, H);
    const int S = seg_plan(s.bv);
    cudaEvent_t a, b;
    OK(cudaEventCreate(&a));
    OK(cudaEventCreate(&b));
    OK(cudaEventRecord(a));
    if (which == 0) {  // one sort pass
      s.set(s.L.counters, TK_SORT, 1);
      radix_pass_kernel<<<dim3(1, s.L.nb_radix), RADIX_BLOCK>>>(s.bv, 0);
    } else if (which == 1) {  // the chunk weights' prefix
      s.set(s.L.counters, TK_CHUNK, 1);
      chunk_kernel<<<dim3(1, s.L.nb_radix), 256>>>(s.bv);
    } else if (which == 2) {  // the row and segment counts' scans
      s.set(s.L.counters, TK_SCAN, 1);
      list_scan_kernel<<<dim3(1, 8), SCAN_THREADS>>>(s.bv, S);
    } else {  // nothing waits: a view already given up on is left alone by every kernel
      s.set(s.L.counters, CI_STATUS, ST_BOUNDS | ST_WAIT);
    }
    OK(cudaGetLastError());
    if (launch_binning_geometry(s.bv, 0)) rc = 1;  // (once a state: the classes' counts start at 0) every later kernel leaves the view alone
    OK(cudaEventRecord(b));
    OK(cudaDeviceSynchronize());
    float ms;
    OK(cudaEventElapsedTime(&ms, a, b));
    std::vector<uint2> ranges(s.L.T());
    OK(cudaMemcpy(ranges.data(), s.geom + s.L.ranges, ranges.size() * 8, cudaMemcpyDeviceToHost));
    bool empty = true;
    for (const uint2 &r : ranges) empty = empty && r.x == r.y;
    printf("%d status %u empty %d ms %.1f\n", which, s.get(s.L.counters, CI_STATUS), (int)empty, ms);
    OK(cudaFree(s.geom));
  }
  return rc;
}
