// Selection of the K nearest from candidate buffers by FP32 squared distances, and the SPH
// sums over them: what the group searches (knn_group.cu, phase_group.cu) share.
#pragma once
#include "knn_wq.cuh"

namespace nbk {
namespace {

constexpr int kGrpSlack = 3;  // entries beyond the K-th a buffer cut may leave
// The reference's lists start with squared distances of kMaxValue and take nothing at or
// beyond it: a query whose K-th bound is not surely below is left to a search with such a list.
constexpr float kGrpFarthest = 0.99999e32f;

// S slots of 32 neighbours: K <= 32 S. Groups shrink as the buffers grow, so that a warp's
// shared memory stays near 6 KB.
template <int S>
struct GrpCfg {
  static constexpr int G = S == 1 ? 8 : (S == 2 ? 4 : 2);
  static constexpr int cap = 64 * S;
};

// The lane index, read once: taken from threadIdx.x it is read again wherever it is used (75
// special-register reads a query).
__device__ __forceinline__ int lane_id() {
  int l;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));
  return l;
}

// Largest of the warp's keys (non-negative doubles' bit patterns).
__device__ __forceinline__ long long warp_max_key(long long k) {
  const unsigned hi = (unsigned)(k >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)k : 0u);
  return (long long)(((unsigned long long)mh << 32) | ml);
}

// Keep threshold for the K-th smallest FP32 squared distance s: every particle whose true
// distance is at most the true K-th has an FP32 squared distance at or below it, and it is
// at or above the true K-th squared distance.
__device__ __forceinline__ float grp_thresh(float s, float two_e) {
  float r;  // within 2^-22 of the square root, inside the 2^-20 margin
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(s));
  const float u = __fmul_ru(r, 1.0f + 1.0f / 1048576.0f);
  const float t = __fadd_ru(u, two_e);
  return __fmul_ru(__fmul_ru(t, t), 1.0f + 1.0f / 1048576.0f);
}

struct GrpCut {
  float thr;   // bound of the cut (-1: FP32 does not resolve the distances, or kGrpFarthest)
  float smin;  // the smallest squared distance
  int cnt;     // entries left
};

// Cut a query's buffer of cnt >= K entries back to those within the bound of its K-th
// smallest (or of one of the `slack` next ones). Not inlined: the kernel's hot loops must
// stay within the instruction cache (inlined everywhere, ten of eleven issue slots waited
// for instructions).
template <int S>
__device__ __noinline__ GrpCut grp_tighten(unsigned* bs, int* bi, int lane, int cnt, int K,
                                           int slack, float two_e) {
  const unsigned FULL = 0xffffffffu;
  constexpr int R = 2 * S;
  GrpCut out;
  unsigned r[R];
  __syncwarp();
  unsigned lo = 0xffffffffu, hi = 0u;
#pragma unroll
  for (int t = 0; t < R; t++) {
    const int p = t * 32 + lane;
    const bool in = p < cnt;
    r[t] = in ? bs[p] : 0xffffffffu;
    lo = min(lo, r[t]);
    if (in) hi = max(hi, r[t]);
  }
  lo = __reduce_min_sync(FULL, lo);
  hi = __reduce_max_sync(FULL, hi);
  out.smin = __uint_as_float(lo);
  out.cnt = cnt;
  // invariant: at least K entries are <= hi; done as soon as K to K + slack are. The first
  // pivot assumes counts growing as the volume, the next ones halve the interval of values
  float pv = __uint_as_float(hi) * (0.3f + 0.7f * __fdividef((float)K, (float)cnt));
#pragma unroll 1
  while (lo < hi && cnt > K + slack) {
    const unsigned mid = max(min(__float_as_uint(pv), hi - 1u), lo);
    int c = 0;
#pragma unroll
    for (int t = 0; t < R; t++) c += __popc(__ballot_sync(FULL, r[t] <= mid));
    if (c >= K) {
      hi = mid;
      if (c <= K + slack) break;
    } else {
      lo = mid + 1;
    }
    // halved before the sum: between squares near FP32's end the pivot would be infinite and
    // each step one unit in the last place
    pv = 0.5f * __uint_as_float(lo) + 0.5f * __uint_as_float(hi);
  }
  unsigned kth = 0u;
#pragma unroll
  for (int t = 0; t < R; t++)
    if (r[t] <= hi) kth = max(kth, r[t]);
  kth = __reduce_max_sync(FULL, kth);
  out.thr = grp_thresh(__uint_as_float(kth), two_e);
  if (kth < 0x0da24260u || !(out.thr <= kGrpFarthest)) {  // below 1e-30, beyond kMaxValue
    out.thr = -1.f;
    return out;
  }
  if (cnt == K) return out;
  const unsigned tb = __float_as_uint(out.thr);
  int id[R], n = 0;
#pragma unroll
  for (int t = 0; t < R; t++) id[t] = bi[t * 32 + lane];
  __syncwarp();
#pragma unroll
  for (int t = 0; t < R; t++) {
    const bool keep = r[t] <= tb;
    const unsigned pm = __ballot_sync(FULL, keep);
    if (keep) {
      const int d = n + __popc(pm & ((1u << lane) - 1u));
      bs[d] = r[t];
      bi[d] = id[t];
    }
    n += __popc(pm);
  }
  __syncwarp();
  out.cnt = n;
  return out;
}

// Ascending sort of the 32 S (key, index) pairs over the warp, position p = s * 32 + lane.
template <int S>
__device__ __forceinline__ void grp_sort(long long key[S], int idx[S], int lane) {
  const unsigned FULL = 0xffffffffu;
#pragma unroll
  for (int size = 2; size <= 32 * S; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= 32) {
        const int ds = stride >> 5;
#pragma unroll
        for (int s = 0; s < S; s++) {
          if (s & ds) continue;
          const bool up = ((s * 32) & size) == 0;
          if ((key[s] > key[s + ds]) == up) {
            const long long k = key[s];
            key[s] = key[s + ds];
            key[s + ds] = k;
            const int i = idx[s];
            idx[s] = idx[s + ds];
            idx[s + ds] = i;
          }
        }
      } else {
#pragma unroll
        for (int s = 0; s < S; s++) {
          const long long ok = __shfl_xor_sync(FULL, key[s], stride);
          const int oj = __shfl_xor_sync(FULL, idx[s], stride);
          const bool up = ((s * 32 + lane) & size) == 0, lower = (lane & stride) == 0;
          if ((lower == up) ? (ok < key[s]) : (ok > key[s])) {
            key[s] = ok;
            idx[s] = oj;
          }
        }
      }
    }
  }
}

// The K smallest of the cnt <= 32 (S + 1) keys (one per lane and slot; index -1: none): the
// largest dropped until K are left, their indices into bi[0 .. K).
template <int S>
__device__ __forceinline__ void grp_keep(long long key[S + 1], int idx[S + 1], int* bi, int lane,
                                         int cnt, int K) {
  const unsigned FULL = 0xffffffffu;
  for (int left = cnt; left > K; left--) {
    long long mx = 0;
#pragma unroll
    for (int s = 0; s <= S; s++) mx = max(mx, key[s]);
    mx = warp_max_key(mx);
    int gone = 0;  // one holder of the largest leaves
#pragma unroll
    for (int s = 0; s <= S; s++) {
      const unsigned b = gone ? 0u : __ballot_sync(FULL, idx[s] >= 0 && key[s] == mx);
      if (b) {
        gone = 1;
        if (lane == __ffs(b) - 1) {
          key[s] = 0;
          idx[s] = -1;
        }
      }
    }
  }
  int n = 0;
  __syncwarp();
#pragma unroll
  for (int s = 0; s <= S; s++) {
    const unsigned pm = __ballot_sync(FULL, idx[s] >= 0);
    if (idx[s] >= 0) bi[n + __popc(pm & ((1u << lane) - 1u))] = idx[s];
    n += __popc(pm);
  }
  __syncwarp();
}

// Sums of the G rows of 32 S doubles, 32 / G lanes a row: on return the first of row q's
// lanes holds its sum.
template <int S>
__device__ __forceinline__ double grp_row_sums(const unsigned (*bs)[GrpCfg<S>::cap], int lane) {
  constexpr int lanes = 32 / GrpCfg<S>::G, per = 32 * S / lanes;
  static_assert((per & (per - 1)) == 0, "the rotation wraps");
  const double* row =
      reinterpret_cast<const double*>(bs[lane / lanes]) + (lane % lanes) * per;
  double acc = 0.0;
#pragma unroll
  for (int t = 0; t < per; t++) acc = dadd(acc, row[(t + lane) & (per - 1)]);
#pragma unroll
  for (int o = 1; o < lanes; o <<= 1) acc = dadd(acc, __shfl_xor_sync(0xffffffffu, acc, o));
  return acc;
}

// Marks in a row of squared distances: the farthest neighbour sits at q = 2 exactly in the
// reference's arithmetic (the table's last entry); no neighbour in this place.
constexpr double kGrpFar = -1.0, kGrpNone = -2.0;

// W of one row entry: u = sqrt(d2) c1 is the table coordinate (c1 = 1 / (h delta)).
__device__ __forceinline__ double grp_w(double d2, double c1, int kr, const double* T) {
  const int hi = __double2hiint(d2);
  if (hi < 0) return d2 == kGrpFar ? T[kr - 1] : 0.0;
  return w_at_u(dmul(sqrt_newton(d2), c1), kr, T);
}

// The symmetric density sums of a group: row q of bs holds query q's squared distances (and
// marks), bi its neighbours; lane q its table scale c1, its own weight wn and wm = wn times
// its mass. rho_q: the queries' densities, rho: all particles' (by index).
template <int S>
__device__ __forceinline__ void grp_sums(unsigned (*bs)[GrpCfg<S>::cap],
                                         const int (*bi)[GrpCfg<S>::cap], const P4* pos,
                                         double* rho_q, double* rho, const double* T, int kr,
                                         int lane, unsigned okm, int K, double c1, double wn,
                                         double wm) {
  const unsigned FULL = 0xffffffffu;
#pragma unroll 1
  for (unsigned left = okm; left; left &= left - 1) {
    const int q = __ffs(left) - 1;
    const double c = __shfl_sync(FULL, c1, q), m = __shfl_sync(FULL, wm, q);
    double* row = reinterpret_cast<double*>(bs[q]);
#pragma unroll
    for (int s = 0; s < S; s++) {
      const int p = s * 32 + lane;
      double t = 0.0;
      if (p < K) {
        const int j = bi[q][p];
        const double wq = grp_w(row[p], c, kr, T);
        atomicAdd(&rho[j], dmul(wq, m));
        t = dmul(wq, pos[j].m);
      }
      row[p] = t;
    }
  }
  __syncwarp();
  const double acc = grp_row_sums<S>(bs, lane);
  constexpr int lanes = 32 / GrpCfg<S>::G;
  const int q = lane / lanes;
  const double n = __shfl_sync(FULL, wn, q);
  if (lane % lanes == 0 && ((okm >> q) & 1u)) atomicAdd(&rho_q[q], dmul(acc, n));
  __syncwarp();
}

}  // namespace
}  // namespace nbk
