// k-nearest-neighbour queries and the SPH quantities built on them: the per-particle
// loops of CalcDensity, CalcVelDensity, CalcDensityParticle and CalcVelDensityParticle
// (KDCalcSmoothQuantities.cxx:203-389, 768-920) and the coordinate forms
// CalcDensityPosition / CalcVelDensityPosition (:1092-1207) as epilogues of the warp-per-query
// search of knn_wq.cuh, points near one another, and the batched density.
#include <algorithm>
#include <map>
#include <mutex>

#include "knn_core.cuh"
#include "knn_wq.cuh"

namespace nbk {

namespace {

// One warp's work of the lane-per-query form: up to 32 queries of one tree (lane = query).
// `qi` indexes the per-query outputs, `self` is the query's tree index (-1 for a point), K the
// heap size. All lanes of the warp call this together.
template <int KMAX, int EPI>
__device__ void run_warp(const KnnArgs& a, const TreeView& tv, WarpSmem<KMAX>& w, int lane,
                         bool valid, int qi, int self, const double x0[3], int K) {
  double top = knn_search<KMAX>(a, tv, w, lane, valid, self, x0, K);
  if (!valid) return;
  if (EPI == kEpiNN) {  // the heap popped into the row, its largest last
    int Kc = K;
    double d;
    int j;
    if (a.drop_largest) {
      heap_pop<KMAX>(w, lane, Kc, d, j);
      Kc--;
    }
    const size_t row = (size_t)qi * a.kout;
    for (int i = a.kout - 1; i >= 0; i--) {
      heap_pop<KMAX>(w, lane, Kc, d, j);
      Kc--;
      a.nn[row + i] = j;
      a.d2[row + i] = d;
    }
    return;
  }
  const int kr = a.kernres;
  const double inv_delta = 0.5 * (double)(kr - 1);  // 1 / table step, exact
  // the heap holds exactly the k neighbours
  for (int s = 0; s < K; s++)
    if (w.hi[s][lane] < 0) {
      atomicExch(a.err, kErrTooFew);
      if (EPI == kEpiSave) a.nn[(size_t)qi * K + K - 1] = -1;  // no row
      return;
    }
  if (EPI == kEpiSave) {  // the farthest, the heap's root, last
    for (int s = 0; s < K; s++) a.nn[(size_t)qi * K + (s == 0 ? K - 1 : s - 1)] = w.hi[s][lane];
    return;
  }
  const double* T = a.kernel;
  if (EPI == kEpiVelPart) {
    // KDCalcSmoothQuantities.cxx:354-383: |dv| of the Nsearch neighbours, keep the
    // Nsmooth smallest, h = 0.5 max, sum Wsm(|dv|/h) h^-3 with unit weights
    const V4 vi = make_v4(a.qv[3 * (size_t)qi], a.qv[3 * (size_t)qi + 1],
                          a.qv[3 * (size_t)qi + 2], 0.0);
    for (int s = 0; s < K; s++) {
      const V4 vj = tv.vel[w.hi[s][lane]];
      w.hd[s][lane] = sqrt_newton(dist2_exact(vi.x, vi.y, vi.z, vj.x, vj.y, vj.z));
    }
    const int ns = min(a.nsmooth, K);
    if (ns < K) {
      // max-heap over the first ns values, then keep the ns smallest of the rest
      for (int s = ns / 2 - 1; s >= 0; s--) {
        const double d = w.hd[s][lane];
        heap_sift<KMAX>(w, lane, ns, s, d, 0);
      }
      for (int s = ns; s < K; s++) {
        const double d = w.hd[s][lane];
        if (dkey(d) < dkey(w.hd[0][lane])) heap_sift<KMAX>(w, lane, ns, 0, d, 0);
      }
    }
    long long vmaxk = 0;
    for (int s = 0; s < ns; s++) vmaxk = max(vmaxk, dkey(w.hd[s][lane]));
    const double ih = recip_newton(0.5 * __longlong_as_double(vmaxk));
    const double norm = dmul(dmul(ih, ih), ih);
    double acc = 0.0;
    for (int s = 0; s < ns; s++) {
      const double vd = w.hd[s][lane];
      const double q = dmul(vd, ih);
      const double wq = dkey(vd) == vmaxk ? T[kr - 1] : wsm_line(q, kr, inv_delta, T);  // q = 2
      acc = dadd(acc, dmul(wq, norm));
    }
    a.vden[qi] = acc;
    return;
  }
  // KDCalcSmoothQuantities.cxx:260-286 (kEpiDensity), :1092-1145 (kEpiDensPart)
  // One reciprocal per query replaces the per-neighbour divisions (r/h and the table
  // step); the density moves by a few units in the last place, far inside 1e-12.
  const double me_m = EPI == kEpiDensPart ? 0.0 : tv.pos[self].m;
  double hh = 0.5 * __dsqrt_rn(top);
  double ih = 1.0 / hh;
  double norm = dmul(dmul(ih, ih), ih);  // 1 / h^3 (the reference takes pow(h, 3))
  double wnorm = EPI == kEpiDensPart ? norm : 0.5 * norm;
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
    if (EPI != kEpiDensPart) atomicAdd(&a.rho[j], dmul(wij, me_m));
  }
  if (EPI == kEpiDensPart) a.rho[qi] = acc;
  else atomicAdd(&a.rho[self], acc);
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
    run_warp<KMAX, kEpiDensity>(a, tv, ws[warp], lane, valid, self, self, x0, K);
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

// ---- points near one another: a lane each

// Points in an order of space with a small k: a warp walks the tree once for 32 of them, where a
// warp per point walks it 32 times for less work each. It pays as long as the walk serves one
// neighbourhood, and a warp takes as long as its slowest point. So a warp takes its points
// together where the box around them, grown by a neighbourhood, is a small multiple of the
// smallest of their neighbourhoods (the node around a point with more than k particles); or
// where all of them lie inside one or two such nodes, if nearly all warps' do (points in tree
// order; a few such warps between others would only be the last to end). The other warps' points
// go to a list that the warp-per-point search serves.
// Measured (density at the points, ms; all warps together, a warp per point, this rule):
// 262,144 points on sightlines among 500,009 particles k = 4 0.46, 1.21, 0.44, k = 12 0.88, 1.40,
// 0.76; in no order k = 8 24, 1.37, 1.25; on a grid k = 8 2.00, 1.24, 1.24 (multiples of 12 and
// 30: 1.47 and 2.00); 0.002 beside particles in tree order k = 8 1.29, 1.20, 1.19; 262,144 of
// 2^20 particles in tree order k = 8 0.88, 1.34, 0.91. 131,072 points in no order: 0.70 a warp
// each, 0.66; on a grid 0.65, 0.67.
constexpr float kPointsVolume = 6.f;
constexpr int kPointsHomes = 2;
// Fewer points leave SMs without warps (65,536 on sightlines, k = 12: 0.35 a warp each, 0.41),
// and the longer the lists, the more there must be to hide a slow warp: k = 16 on sightlines and
// beside particles in tree order, 131,072 points 0.71 and 0.69 a warp each, 0.55 and 0.89;
// 262,144 1.42 and 1.30, 0.91 and 1.38; 2^20 5.46 and 5.13, 2.29 and 4.77; k = 24, 262,144 1.61
// and 1.47, 1.28 and 1.68.
constexpr int kPointsK = 16, kPointsMin = 1 << 19;
constexpr int kPointsShortK = 12, kPointsShortMin = kPointsSmallest;

inline bool points_share_warps(const KnnArgs& a) {
  return a.qmode == 1 && a.fb &&
         ((a.kheap <= kPointsShortK && a.nq >= kPointsShortMin) ||
          (a.kheap <= kPointsK && a.nq >= kPointsMin));
}

// a.fb here: [0] warps on the list, [1] fours of points taken from it, [2] warps in tree order;
// then per warp what it may do (1: one neighbourhood, 2: tree order), then the list.
__global__ void __launch_bounds__(256) k_points_class(KnnArgs a) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, gw = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (gw * 32 >= a.nq) return;
  const TreeView& tv = a.tv;
  const size_t at = 3 * (size_t)min(gw * 32 + lane, a.nq - 1);
  const double x[3] = {a.qx[at], a.qx[at + 1], a.qx[at + 2]};
  int h, start, size;
  wq_home_point(tv, x, a.kheap + 1, h, start, size);
  const NodeRec r = tv.node[tv.nbase + h];
  float vol = 1.f;
  bool inside = true;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const float c = __double2float_rn(x[d]);
    inside = inside && c >= r.lo[d] && c <= r.hi[d];
    float lo = c, hi = c;
    for (int o = 16; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(FULL, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, o));
    }
    const float e = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(r.hi[d] - r.lo[d])));
    vol *= (hi - lo) / e + 1.f;
  }
  const unsigned same = __match_any_sync(FULL, h);
  const bool ordered = __all_sync(FULL, inside) &&
                       __popc(__ballot_sync(FULL, lane == __ffs(same) - 1)) <= kPointsHomes;
  if (lane != 0) return;
  a.fb[3 + gw] = (vol <= kPointsVolume ? 1 : 0) | (ordered ? 2 : 0);  // (NaN: not below)
  if (ordered) atomicAdd(&a.fb[2], 1);
}

template <int KMAX, int EPI>
__global__ void __launch_bounds__(32 * warps_per_block<KMAX>()) k_knn_points(KnnArgs a) {
  constexpr int WPB = warps_per_block<KMAX>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  WarpSmem<KMAX>* ws = reinterpret_cast<WarpSmem<KMAX>*>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gw = blockIdx.x * WPB + warp, qi = gw * 32 + lane;
  if (gw * 32 >= a.nq) return;
  const int warps = (a.nq + 31) / 32;
  const int what = a.fb[3 + gw];
  if (!(what & 1) && !(what && a.fb[2] >= warps - warps / 8)) {
    if (lane == 0) a.fb[3 + warps + atomicAdd(&a.fb[0], 1)] = gw;
    return;
  }
  const bool valid = qi < a.nq;
  const size_t at = 3 * (size_t)(valid ? qi : gw * 32);
  const double x0[3] = {a.qx[at], a.qx[at + 1], a.qx[at + 2]};
  run_warp<KMAX, EPI>(a, a.tv, ws[warp], lane, valid, qi, -1, x0, a.kheap);
}

// The points of the listed warps, a warp each: a persistent grid whose warps pull four at a
// time.
template <int EPI>
__global__ void __launch_bounds__(32 * kWqWpb, 4) k_knn_points_list(KnnArgs a) {
  __shared__ WqSmem ws[kWqWpb];
  const unsigned FULL = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int count = 8 * a.fb[0], *list = a.fb + 3 + (a.nq + 31) / 32;
  for (int guard = 0; guard <= count; guard++) {
    int i = 0;
    if (lane == 0) i = atomicAdd(&a.fb[1], 1);
    i = __shfl_sync(FULL, i, 0);
    if (i >= count) return;
    const int q0 = list[i >> 3] * 32 + (i & 7) * 4;
#pragma unroll 1
    for (int qi = q0; qi < min(q0 + 4, a.nq); qi++) {
      const double* x = a.qx + 3 * (size_t)qi;
      const double x0[3] = {x[0], x[1], x[2]};
      wq_run<1, EPI>(a, a.tv, ws[warp], lane, qi, -1, x0, a.kheap);
      __syncwarp();
    }
  }
}

template <int KMAX, int EPI>
int launch_points(const KnnArgs& a, cudaStream_t st) {
  constexpr int WPB = warps_per_block<KMAX>();
  const size_t sm = sizeof(WarpSmem<KMAX>) * WPB;
  NBK_TRY(ensure_dyn_smem((const void*)k_knn_points<KMAX, EPI>, (int)sm));
  int nsm = 0, dev = 0;
  NBK_CUDA_TRY(cudaGetDevice(&dev));
  NBK_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  NBK_CUDA_TRY(cudaMemsetAsync(a.fb, 0, 3 * sizeof(int), st));
  Phase ph("knn_points", st);
  const unsigned warps = ((unsigned)a.nq + 31) / 32;
  k_points_class<<<(warps + 7) / 8, 256, 0, st>>>(a); note_launch();
  k_knn_points<KMAX, EPI><<<(warps + WPB - 1) / WPB, 32 * WPB, sm, st>>>(a); note_launch();
  k_knn_points_list<EPI><<<(unsigned)(4 * nsm), 32 * kWqWpb, 0, st>>>(a); note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  return NBK_OK;
}

template <int EPI>
int launch_e(const KnnArgs& a, cudaStream_t st) {
  if (EPI != kEpiDensPart && EPI != kEpiVelPart && a.fb && group_search_serves(a, EPI))
    return launch_knn_group(a, EPI, st);
  if constexpr (EPI == kEpiNN || EPI == kEpiDensPart || EPI == kEpiVelPart || EPI == kEpiSave) {
    if (points_share_warps(a)) return launch_points<kPointsK, EPI>(a, st);
  }
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
