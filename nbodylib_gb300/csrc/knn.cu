// k-nearest-neighbour queries and the SPH quantities built on them: the per-particle
// loops of CalcDensity, CalcVelDensity, CalcDensityParticle and CalcVelDensityParticle
// (KDCalcSmoothQuantities.cxx:203-389, 768-920) and the coordinate forms
// CalcDensityPosition / CalcVelDensityPosition (:1092-1207) as epilogues of the warp-per-query
// search of knn_wq.cuh, and the batched density.
#include <algorithm>
#include <map>
#include <mutex>

#include "knn_core.cuh"
#include "knn_wq.cuh"

namespace nbk {

namespace {

// One warp's work of the batched density's lane-per-query form: up to 32 queries of one tree
// (lane = query); `self` is the query's tree index, K the heap size. All lanes of the warp
// call this together.
template <int KMAX>
__device__ void run_warp(const KnnArgs& a, const TreeView& tv, WarpSmem<KMAX>& w, int lane,
                         bool valid, int self, const double x0[3], int K) {
  double top = knn_search<KMAX>(a, tv, w, lane, valid, self, x0, K);
  if (!valid) return;
  const int kr = a.kernres;
  const double inv_delta = 0.5 * (double)(kr - 1);  // 1 / table step, exact
  // the heap holds exactly the k neighbours (target search)
  for (int s = 0; s < K; s++)
    if (w.hi[s][lane] < 0) {
      atomicExch(a.err, kErrTooFew);
      return;
    }
  const double* T = a.kernel;
  const P4 me = tv.pos[self];
  // KDCalcSmoothQuantities.cxx:260-286
  // One reciprocal per query replaces the per-neighbour divisions (r/h and the table
  // step); the density moves by a few units in the last place, far inside 1e-12.
  double hh = 0.5 * __dsqrt_rn(top);
  double ih = 1.0 / hh;
  double norm = dmul(dmul(ih, ih), ih);  // 1 / h^3 (the reference takes pow(h, 3))
  double wnorm = 0.5 * norm;
  double acc = 0.0;
  const long long topk = dkey(top);
  for (int s = 0; s < K; s++) {
    double d2 = w.hd[s][lane];
    int j = w.hi[s][lane];
    // the farthest neighbour sits at q = 2 exactly in the reference's arithmetic (the
    // table's last entry, 0 for the compact kernels); the product with 1/h could land
    // an ulp below it, in the previous cell
    double q = dmul(sqrt_newton(d2), ih);
    double wq = dkey(d2) == topk ? T[kr - 1] : wsm_line(q, kr, inv_delta, T);
    double wij = dmul(wq, wnorm);
    acc = dadd(acc, dmul(wij, tv.pos[j].m));
    atomicAdd(&a.rho[j], dmul(wij, me.m));
  }
  atomicAdd(&a.rho[self], acc);
}

// Batched density: a persistent grid whose warps pull (tree, query bucket) work items
// from an atomic counter until the list is exhausted; every tree is searched with its
// own k = min(k, n_tree - 1). The loop is bounded by the item count.
template <int KMAX>
__global__ void __launch_bounds__(32 * warps_per_block<KMAX>()) k_knn_batch(KnnArgs a, BatchArgs b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WarpSmem<KMAX>* ws = reinterpret_cast<WarpSmem<KMAX>*>(smem_raw);
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int guard = 0; guard < b.nitems + 1; guard++) {
    int item = 0;
    if (lane == 0) item = atomicAdd(b.counter, 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= b.nitems) break;
    WorkItem it = b.items[item];
    TreeInfo ti = b.trees[it.tree];
    TreeView tv = a.tv;
    tv.n = ti.n;
    tv.pstart = ti.pstart;
    tv.nbase = ti.nbase;
    int K = min(a.kheap, ti.n - 1);
    if (K < 1) continue;
    bool valid = lane < it.count;
    int self = ti.pstart + it.q0 + (valid ? lane : 0);
    P4 p = tv.pos[self];
    double x0[3] = {p.x, p.y, p.z};
    run_warp<KMAX>(a, tv, ws[warp], lane, valid, self, x0, K);
    __syncwarp();
  }
}

// ---- warp per query (knn_wq.cuh): target queries

// 64 registers per thread (4 blocks of 8 warps per SM): the occupancy outweighs the few
// spills of the two- and four-slot lists (measured at 2^20 and 2^22 clustered particles)
template <int S, int EPI>
__global__ void __launch_bounds__(32 * kWqWpb, 4) k_knn_wq(KnnArgs a) {
  __shared__ WqSmem ws[kWqWpb];
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int qi = blockIdx.x * kWqWpb + warp;
  if (qi >= a.nq) return;
  const TreeView& tv = a.tv;
  int self = -1;
  double x0[3];
  if (a.qmode == 1) {
#pragma unroll
    for (int d = 0; d < 3; d++) x0[d] = a.qx[3 * (size_t)qi + d];
  } else {
    self = a.qmode == 0 ? a.q0 + qi : a.qidx[qi];
    if (a.qmode == 2 && (self < 0 || self >= tv.n)) {  // device-resident targets: checked here
      if (lane == 0) atomicExch(a.err, kErrTarget);
      return;
    }
    P4 p = tv.pos[self];
    x0[0] = p.x;
    x0[1] = p.y;
    x0[2] = p.z;
  }
  wq_run<S, EPI>(a, tv, ws[warp], lane, qi, self, x0, a.kheap);
}

template <int S, int EPI>
int launch_wq(const KnnArgs& a, cudaStream_t st) {
  unsigned blocks = (unsigned)((a.nq + kWqWpb - 1) / kWqWpb);
  if (blocks == 0) return NBK_OK;
  static const char* kNames[] = {"knn_nn", "knn_density", "knn_density_veldensity", "knn_veldensity",
                                 "knn_density_particle", "knn_veldensity_particle", "knn_density_save",
                                 "knn_save"};
  Phase ph(kNames[EPI], st);
  k_knn_wq<S, EPI><<<blocks, 32 * kWqWpb, 0, st>>>(a); note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  return NBK_OK;
}

template <int EPI>
int launch_e(const KnnArgs& a, cudaStream_t st) {
  if (EPI != kEpiDensPart && EPI != kEpiVelPart && group_search_serves(a))
    return launch_knn_group(a, EPI, st);
  if (a.kheap <= 32) return launch_wq<1, EPI>(a, st);
  if (a.kheap <= 64) return launch_wq<2, EPI>(a, st);
  if (a.kheap <= 128) return launch_wq<4, EPI>(a, st);
  set_error("k larger than 127 is not supported by the GPU kNN kernels");
  return NBK_ERR_UNSUPPORTED;
}

template <int KMAX>
int launch_batch_t(const KnnArgs& a, const BatchArgs& b, cudaStream_t st) {
  constexpr int WPB = warps_per_block<KMAX>();
  size_t sm = sizeof(WarpSmem<KMAX>) * WPB;
  // persistent grid: every resident block of this device (cached per device)
  static std::mutex mu;
  static std::map<int, int> grids;
  int dev = 0, grid = 0;
  NBK_CUDA_TRY(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = grids.find(dev);
    if (it != grids.end()) grid = it->second;
  }
  if (grid == 0) {
    NBK_TRY(ensure_dyn_smem((const void*)k_knn_batch<KMAX>, (int)sm));
    int nsm = 0, per = 0;
    NBK_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    NBK_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_knn_batch<KMAX>, 32 * WPB, sm));
    grid = nsm * (per > 0 ? per : 1);
    std::lock_guard<std::mutex> lk(mu);
    grids[dev] = grid;
  }
  int blocks = std::min(grid, (b.nitems + WPB - 1) / WPB);
  if (blocks <= 0) return NBK_OK;
  Phase ph("knn_density_batch", st);
  k_knn_batch<KMAX><<<blocks, 32 * WPB, sm, st>>>(a, b); note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  return NBK_OK;
}

}  // namespace

int launch_knn_batch(const KnnArgs& a, const BatchArgs& b, cudaStream_t st) {
  if (b.warp_per_query && a.kheap <= 128) return launch_knn_group_batch(a, b, st);
  if (a.kheap <= 16) return launch_batch_t<16>(a, b, st);
  if (a.kheap <= 33) return launch_batch_t<33>(a, b, st);
  if (a.kheap <= 65) return launch_batch_t<65>(a, b, st);
  if (a.kheap <= 128) return launch_batch_t<128>(a, b, st);
  set_error("k larger than 127 is not supported by the GPU kNN kernels");
  return NBK_ERR_UNSUPPORTED;
}

int launch_knn(const KnnArgs& a, int epi, cudaStream_t st) {
  switch (epi) {
    case kEpiNN: return launch_e<kEpiNN>(a, st);
    case kEpiDensity: return launch_e<kEpiDensity>(a, st);
    case kEpiDensVel: return launch_e<kEpiDensVel>(a, st);
    case kEpiVel: return launch_e<kEpiVel>(a, st);
    case kEpiDensPart: return launch_e<kEpiDensPart>(a, st);
    case kEpiVelPart: return launch_e<kEpiVelPart>(a, st);
    case kEpiDensSave: return launch_e<kEpiDensSave>(a, st);
    case kEpiSave: return launch_e<kEpiSave>(a, st);
  }
  set_error("unknown kNN epilogue");
  return NBK_ERR_INVALID;
}

}  // namespace nbk
