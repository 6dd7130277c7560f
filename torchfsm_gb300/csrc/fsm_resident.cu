// Choice and launch of the resident 2D kernels (fsm_resident.cuh).
#include <math.h>
#include <string.h>

#include <map>
#include <mutex>
#include <tuple>

#include "fsm_resident.cuh"

namespace fsm {

namespace {

constexpr size_t kSmemMax = 227 * 1024;   // per CTA
constexpr size_t kSmemHalf = 114 * 1024;  // above this one CTA fits per SM
// Steps of one launch: long runs return to the stream now and then. A batch that fills the device returns
// sooner, so that a stream of higher priority finds SMs after some milliseconds (2048 steps of 64^2 x 1000
// hold them for 0.1 s at a time). A launch loads and stores its samples' state and tables: 64^2 x 1000 183.9 -> 184.1
// us per step, Burgers 128^2 x 30 59.5 -> 59.8.
constexpr int kResidentSteps = 2048;
constexpr int kResidentStepsFull = 256;

ResKernel kernel_of(const FsmPlan* p) {
  switch (p->nl) {
    case FSM_NL_VORTICITY: return resident_vorticity(p->n[0], p->n[1]);
    case FSM_NL_CONVECTION: return resident_convection(p->n[0], p->n[1]);
    case FSM_NL_LERAY: return resident_leray(p->n[0], p->n[1]);
  }
  return {};
}

void fill(cudaLaunchConfig_t& lc, cudaLaunchAttribute& at, const ResConfig& c, size_t smem, int batch, cudaStream_t st) {
  memset(&lc, 0, sizeof(lc));
  memset(&at, 0, sizeof(at));
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)c.cl;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  lc.gridDim = dim3((unsigned)(batch * c.cl));
  lc.blockDim = dim3((unsigned)c.threads);
  lc.dynamicSmemBytes = smem;
  lc.stream = st;
  lc.attrs = &at;
  lc.numAttrs = 1;
}

// Clusters of this shape that the device holds at once (0: none, or the query failed). The answers
// are kept per (kernel, device, shape): they do not change while the process runs.
int active_clusters(const ResKernel& k, const ResConfig& c, size_t smem) {
  static std::mutex m;
  static std::map<std::tuple<const void*, int, int, int, size_t>, int> known;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const auto key = std::make_tuple((const void*)k.fn, dev, c.cl, c.threads, smem);
  std::lock_guard<std::mutex> lock(m);
  auto it = known.find(key);
  if (it != known.end()) return it->second;
  int n = 0;
  cudaLaunchConfig_t lc;
  cudaLaunchAttribute at;
  fill(lc, at, c, smem, 1, nullptr);
  if (cudaFuncSetAttribute(k.fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, k.fn, &lc) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  known[key] = n;
  return n;
}

}  // namespace

// Cluster size and the choice against the passes, from measurements on GB300 (us per step).
// One wave of clusters takes about A (1 + work / cl), with A set by the transform lengths and work
// by the grid's points (vorticity 64^2: cl 16 / 8 / 4 / 2 / 1: 12.0 / 11.5 / 12.6 / 16.7 / 27; 128^2:
// cl 16 / 12 / 8 / 6 / 5: 23.5 / 24.0 / 26.5 / 29.9 / 32.4); CTAs that share an SM cost about 0.3 of a
// wave each (64^2 x 16: cl 8 on shared SMs 14.2, cl 6 alone 12.3). So the largest cluster that runs
// the batch in one wave alone on its SMs wins, and waves and sharing are weighed with the same sum.
// Groups share a column's inverse transforms while a CTA stays within 192 lanes of columns.
// Against the passes (resident / passes): 64^2 vorticity 1 sample 12.2 / 66, 150: 27 / 83, 1000: 185 /
// 275; 128^2 16: 30 / 108, 128: 152 / 191, 256: 298 / 254; 256^2 7: 39 / 97, 14: 76 / 105, 24: 150 / 134;
// 128x256 velocity 9: 49 / 170. Above 8192 points the passes win once est x points exceeds 190e3, and sooner
// where the batch runs in parts (`parts` above 1: medium batches of 16 steps or more, large ones), resident /
// parts: vorticity 128^2 x 80 (est 4.9) 105 / 105, x 100 (5.4) 117 / 111, x 200 (10.8) 231 / 154; Burgers 128^2 x 80
// (4.9) 119 / 120, x 100 (6.6) 158 / 133; at 32768 points sooner still: 128x256 x 24 (2.9) 80 / 84, x 32 (4.4)
// 117 / 96, vorticity 256x128 x 24 (2.9) 71 / 83, x 32 (4.4) 104 / 98. The Leray projection's passes carry both
// channels in one chain: 128^2 x 100 (6.6) takes 1.2 times as long in parts as here.
bool resident_config(const FsmPlan* p, int batch, int parts, ResConfig* out) {
  const int nx = p->n[0], ny = p->n[1], h = p->h, hk = p->hk;
  if (p->path != 2 || p->integ != FSM_SETDRK4 || batch < 1 || hk != ny / 3 + 1) return false;
  const ResKernel k = kernel_of(p);
  if (!k.fn) return false;
  const int per = p->nl == FSM_NL_CONVECTION ? 2 : 1;       // column items per column
  const int fields = p->nl == FSM_NL_VORTICITY ? 4 : 2;  // fields an item transforms
  const double work = 1.6 * sqrt((double)nx * ny) / 64.0;
  double best = 0.0;
  static const int sizes[] = {16, 12, 10, 8, 6, 5, 4, 3, 2, 1};
  for (int cl : sizes) {
    if (cl > nx / 2) continue;
    ResConfig c;
    c.cl = cl;
    c.rpc = (nx + 2 * cl - 1) / (2 * cl) * 2;
    c.ka = (hk + cl - 1) / cl;
    c.kb = (h - hk + cl - 1) / cl;
    c.pc = (c.ka + c.kb) | 1;
    const int lanes = (c.ka + c.kb) * per * k.tx;
    c.fs = 1;
    while (c.fs < fields && lanes * c.fs * 2 <= 192) c.fs *= 2;
    int t = lanes * c.fs > c.rpc * k.ty ? lanes * c.fs : c.rpc * k.ty;
    t = (t + 31) & ~31;
    c.threads = t > kResThreads ? kResThreads : t;
    c.tables = true;
    c.smem = k.smem(c.rpc, c.ka, c.kb, c.pc, c.fs, p->lin_ch, true, c.threads);
    if (c.smem > kSmemMax) {
      c.tables = false;
      c.smem = k.smem(c.rpc, c.ka, c.kb, c.pc, c.fs, p->lin_ch, false, c.threads);
    }
    if (c.smem > kSmemMax) continue;
    const int cap = active_clusters(k, c, c.smem);
    const int cap1 = c.smem > kSmemHalf ? cap : active_clusters(k, c, kSmemHalf + 1024);
    if (cap < 1 || cap1 < 1) continue;
    const int waves = (batch + cap - 1) / cap;
    const int shared = batch >= cap ? (cap + cap1 - 1) / cap1 : (batch + cap1 - 1) / cap1;  // CTAs per SM
    const double est = waves * (1.0 + work / cl) * (1.0 + 0.3 * (shared - 1));
    if (best == 0.0 || est < best) {
      best = est;
      c.steps = batch < cap ? kResidentSteps : kResidentStepsFull;
      *out = c;
    }
  }
  const double points = (double)nx * ny;
  const bool parted = parts > 1 && p->nl != FSM_NL_LERAY;
  const double line = points > 16384.0 ? 4.2 : 5.0;
  return best > 0.0 && (points <= 8192.0 || (best * points <= 190e3 && !(parted && best > line)));
}

int launch_resident(const FsmPlan* p, const ResConfig& c, const StepArgs& a, cudaStream_t st) {
  const ResKernel k = kernel_of(p);
  cudaLaunchConfig_t lc;
  cudaLaunchAttribute at;
  fill(lc, at, c, c.smem, a.B, st);
  ResArgs r;
  r.a = a;
  r.ka = c.ka;
  r.kb = c.kb;
  r.pc = c.pc;
  r.fs = c.fs;
  r.rpc = c.rpc;
  r.tables = c.tables;
  return cuda_check(cudaLaunchKernelEx(&lc, k.fn, r), "k_plane_resident");
}

}  // namespace fsm
