// Warp-per-query k-nearest-neighbour search: the kNN behind CalcDensityParticle,
// CalcVelDensityParticle, FindNearest / FindNearestPos of given tree particles, the coordinate
// forms (FindNearest(x), CalcDensityPosition, CalcVelDensityPosition) but for points near one
// another with a small k (k_knn_points, knn.cu), and the queries that the group search
// (knn_group.cu) leaves. A warp for any 32 consecutive points walked the tree for all of them at
// once: with points in no spatial order every lane's neighbourhood was opened for the whole warp
// (250,007 points, k = 40, in 500,009 particles: 145 ms; a warp a point does not depend on their
// order).
//
// Replaces the depth-first search of SplitNode/LeafNode::FindNearestPos(target)
// (src/KDTree/KDSplitNode.cxx:15-41, KDLeafNode.cxx:15-28) with its bounded max-heap
// (src/KDTree/PriorityQueue.h:14-85), and the periodic wrapper of KDSplitNode.cxx:1119-1147.
//
// Work mapping: one warp serves one query. The query's k-list is distributed over the
// warp's registers, sorted: position p = s * 32 + lane holds the p-th smallest (d2, index)
// in slot s of that lane (S slots, k <= 32 S). A batch of candidates enters by a bitonic
// sort over the lanes and a merge with the list (one or two slots), or one candidate at a time
// by a ballot (its position) and a shuffle of the tail one place up; the k-th distance
// (the heap top of the reference) is one shuffle away.
//
// Search order: the query's own subtree first -- the smallest node on its path holding
// more than k particles, found from the tree's split rule by integer arithmetic (left
// child = the first (size - 1) / 2 + 1 particles, leaf when size <= b). An FP32 upper
// bound of the k-th distance over that subtree's particles is found first, then they are
// tested; then the rest of the tree -- the subtrees of the siblings of that node and of
// each of its ancestors -- frontier-parallel: each step pops up to 32 stack nodes, one per
// lane, and prunes them against the k-th distance.
//
// FP64 work: candidates are screened by an FP32 lower bound of their squared distance
// (directed rounding, never below the FP64 value); those that pass are compacted into a
// per-warp queue, and the exact FP64 distance ((dx*dx + dy*dy) + dz*dz), the reference's
// association, is computed 32 queued candidates at a time, so the FP64 instructions run
// with every lane busy. A candidate enters when d2 < the k-th distance (strict, as the
// reference's `dist2 < pq->TopPriority()`); the FP32 screen uses a bound at or above the
// k-th distance, the exact test the current k-th distance, so the result is the exact k
// nearest.
#pragma once
#include "nbk_build.h"

namespace nbk {
namespace {

constexpr int kWqStack = 192;      // frontier stack (node indices) per warp
constexpr int kWqBatchLimit = 96;  // above this many entries the stack pops one at a time
constexpr long long kWqSent = 0x7fffffffffffffffll;  // key beyond position k - 1

struct WqSmem {
  int stk[kWqStack];
  int queue[64];        // candidates (tree indices) that passed the FP32 screen
};

// The sorted k-list of one query: keys are the bit patterns of the non-negative squared
// distances (they order as the values do, on the integer pipe).
template <int S>
struct WqList {
  long long key[S];
  int idx[S];
};

template <int S>
__device__ __forceinline__ void wq_init(WqList<S>& L, int lane, int K) {
  const long long kmax = __double_as_longlong(kMaxValue);
#pragma unroll
  for (int s = 0; s < S; s++) {
    int p = s * 32 + lane;
    L.key[s] = p < K ? kmax : kWqSent;  // the reference pre-fills with (-1, MAXVALUE)
    L.idx[s] = -1;
  }
}

// Key at position p of the list (every lane gets it).
template <int S>
__device__ __forceinline__ long long wq_key_at(const WqList<S>& L, int p) {
  long long v = L.key[0];
#pragma unroll
  for (int s = 1; s < S; s++)
    if ((p >> 5) == s) v = L.key[s];
  return __shfl_sync(0xffffffffu, v, p & 31);
}

// Insert (k, j) (the same on every lane) into a list of K entries; the caller has
// checked k < the key at position K - 1.
template <int S>
__device__ __forceinline__ void wq_insert(WqList<S>& L, int lane, int K, long long k, int j) {
  const unsigned FULL = 0xffffffffu;
  int pos = 0;
#pragma unroll
  for (int s = 0; s < S; s++) pos += __popc(__ballot_sync(FULL, L.key[s] <= k));
#pragma unroll
  for (int s = S - 1; s >= 0; s--) {
    long long up = __shfl_up_sync(FULL, L.key[s], 1);
    int upi = __shfl_up_sync(FULL, L.idx[s], 1);
    if (s > 0) {
      long long c = __shfl_sync(FULL, L.key[s - 1], 31);
      int ci = __shfl_sync(FULL, L.idx[s - 1], 31);
      if (lane == 0) {
        up = c;
        upi = ci;
      }
    }
    int p = s * 32 + lane;
    if (p == pos) {
      L.key[s] = k;
      L.idx[s] = j;
    } else if (p > pos) {
      L.key[s] = up;
      L.idx[s] = upi;
    }
    if (p >= K) {
      L.key[s] = kWqSent;
      L.idx[s] = -1;
    }
  }
}

// Ascending bitonic sort of one (key, index) pair per lane over the warp (equal keys are
// never exchanged).
__device__ __forceinline__ void warp_sort_asc(long long& k, int& j, int lane) {
  const unsigned FULL = 0xffffffffu;
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      long long ok = __shfl_xor_sync(FULL, k, stride);
      int oj = __shfl_xor_sync(FULL, j, stride);
      bool up = (lane & size) == 0;
      bool lower = (lane & stride) == 0;
      bool take = (lower == up) ? (ok < k) : (ok > k);
      if (take) {
        k = ok;
        j = oj;
      }
    }
  }
}

// Merge a batch sorted ascending over the lanes into a one-slot list of K <= 32 entries:
// the lower half of Batcher's merge (list ascending against the batch reversed; the list
// keeps ties) holds the 32 smallest of both as a bitonic sequence, which five
// half-cleaners sort.
__device__ __forceinline__ void wq_merge1(WqList<1>& L, int lane, int K, long long k, int j) {
  const unsigned FULL = 0xffffffffu;
  long long rk = __shfl_sync(FULL, k, 31 - lane);
  int rj = __shfl_sync(FULL, j, 31 - lane);
  bool tb = rk < L.key[0];
  long long mk = tb ? rk : L.key[0];
  int mj = tb ? rj : L.idx[0];
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    long long ok = __shfl_xor_sync(FULL, mk, stride);
    int oj = __shfl_xor_sync(FULL, mj, stride);
    bool lower = (lane & stride) == 0;
    bool take = lower ? (ok < mk) : (ok > mk);
    if (take) {
      mk = ok;
      mj = oj;
    }
  }
  if (lane >= K) {
    mk = kWqSent;
    mj = -1;
  }
  L.key[0] = mk;
  L.idx[0] = mj;
}

// The same for a two-slot list of K <= 64 entries (positions 0-31 in slot 0, 32-63 in
// slot 1): against the 128-sequence list ascending ++ (batch padded to 64 with +inf)
// reversed, the lower half keeps slot 0 and takes min(slot 1, batch reversed); that
// bitonic 64-sequence is sorted by an in-lane compare-exchange (stride 32) and five
// shuffle half-cleaners per slot.
__device__ __forceinline__ void wq_merge2(WqList<2>& L, int lane, int K, long long k, int j) {
  const unsigned FULL = 0xffffffffu;
  long long rk = __shfl_sync(FULL, k, 31 - lane);
  int rj = __shfl_sync(FULL, j, 31 - lane);
  long long a0 = L.key[0], a1 = L.key[1];
  int i0 = L.idx[0], i1 = L.idx[1];
  if (rk < a1) {
    a1 = rk;
    i1 = rj;
  }
  if (a1 < a0) {
    long long tk = a0;
    a0 = a1;
    a1 = tk;
    int ti = i0;
    i0 = i1;
    i1 = ti;
  }
#pragma unroll
  for (int stride = 16; stride > 0; stride >>= 1) {
    bool lower = (lane & stride) == 0;
    long long o0 = __shfl_xor_sync(FULL, a0, stride);
    int p0 = __shfl_xor_sync(FULL, i0, stride);
    long long o1 = __shfl_xor_sync(FULL, a1, stride);
    int p1 = __shfl_xor_sync(FULL, i1, stride);
    if (lower ? (o0 < a0) : (o0 > a0)) {
      a0 = o0;
      i0 = p0;
    }
    if (lower ? (o1 < a1) : (o1 > a1)) {
      a1 = o1;
      i1 = p1;
    }
  }
  if (lane >= K) {
    a0 = kWqSent;
    i0 = -1;
  }
  if (32 + lane >= K) {
    a1 = kWqSent;
    i1 = -1;
  }
  L.key[0] = a0;
  L.idx[0] = i0;
  L.key[1] = a1;
  L.idx[1] = i1;
}

// Per-warp search state of one query.
template <int S>
struct WqQuery {
  WqList<S> L;
  int K;
  long long topk;  // key at position K - 1
  float thr;       // FP32 value at or above the k-th distance (screens boxes, particles)
  double xq[3];    // the query point of this pass (exact)
  float qx, qy, qz, eps, two_eps;
  int self;        // tree index excluded by the target search (-1: none)
  int qn;          // candidates waiting in the queue
};

template <int S>
__device__ __forceinline__ void wq_set_point(WqQuery<S>& Q, const TreeView& tv, const double x[3]) {
  Q.xq[0] = x[0];
  Q.xq[1] = x[1];
  Q.xq[2] = x[2];
  Q.qx = __double2float_rn(x[0]);
  Q.qy = __double2float_rn(x[1]);
  Q.qz = __double2float_rn(x[2]);
  Q.eps = query_eps(tv, x[0], x[1], x[2]);
  Q.two_eps = __fadd_ru(Q.eps, tv.eps);
}

// Exact FP64 test of the first `cnt` queued candidates (one per lane) and insertion of
// those below the k-th distance.
template <int S>
__device__ __forceinline__ void wq_flush(WqQuery<S>& Q, WqSmem& w, const TreeView& tv, int lane, int cnt) {
  const unsigned FULL = 0xffffffffu;
  bool have = lane < cnt;
  int ti = have ? w.queue[lane] : 0;
  long long dk = kWqSent;
  if (have) {
    P4 c = tv.pos[ti];
    double d2 = dist2_exact(Q.xq[0], Q.xq[1], Q.xq[2], c.x, c.y, c.z);
    dk = dkey(d2);
    if (Q.self >= 0 && (ti == Q.self || dk == 0)) dk = kWqSent;  // KDLeafNode.cxx:19-21
  }
  unsigned acc = __ballot_sync(FULL, dk < Q.topk);
  if (S <= 2 && __popc(acc) > 2) {
    // many at once: sort the batch and merge it (the k smallest of list and batch: the
    // same entries the one-by-one strict insertions keep, up to exact ties)
    long long k = dk < Q.topk ? dk : kWqSent;
    int j = ti;
    warp_sort_asc(k, j, lane);
    if (S == 1) wq_merge1(*reinterpret_cast<WqList<1>*>(&Q.L), lane, Q.K, k, j);
    else wq_merge2(*reinterpret_cast<WqList<2>*>(&Q.L), lane, Q.K, k, j);
    Q.topk = wq_key_at<S>(Q.L, Q.K - 1);
    acc = 0;
  }
  while (acc) {
    int src = __ffs(acc) - 1;
    acc &= acc - 1;
    long long k = __shfl_sync(FULL, dk, src);
    int j = __shfl_sync(FULL, ti, src);
    if (k < Q.topk) {  // d2 < top, against the k-th distance of this moment
      wq_insert<S>(Q.L, lane, Q.K, k, j);
      Q.topk = wq_key_at<S>(Q.L, Q.K - 1);
    }
  }
  Q.thr = fminf(Q.thr, thresh_hi_bits(Q.topk));
}

// One pass over the tree: the particles [r0, r1) of the subtree at heap index `home` (those
// around the query), then the subtrees of the siblings of home and of each of its ancestors,
// which are tested together, one per lane, instead of descending from the root one level per
// step; or the whole tree when `home` is -1. Frontier-parallel: up to 32 nodes per step are
// tested against the k-th distance. Candidates (32 particles of the range, or the particles of
// two leaves, 16 each, per step) that pass the FP32 screen join the queue, which is flushed 32
// at a time. There is one place each for screening, flushing and testing nodes: inlined
// several times over, the kernels waited for instructions (five of ten issue slots). Returns
// false when the stack would overflow (the caller sets the error word).
template <int S>
__device__ __forceinline__ bool wq_pass(WqQuery<S>& Q, WqSmem& w, const TreeView& tv, int lane,
                                        int home, int r0, int r1) {
  const unsigned FULL = 0xffffffffu;
  int sp = 0, m = 1, h = 0;
  if (home >= 0) {
    m = 31 - __clz(home + 1);  // home's level (at most 31, n < 2^31)
    if (lane < m) {
      const int a = ((home + 1) >> lane) - 1;
      h = (a & 1) ? a + 1 : a - 1;
    }
  }
  unsigned lm = 0;     // leaves of the last step not screened yet (a bit per lane)
  NodeRec r{};
  int st = 0, ct = 0;  // the leaf this half warp screens, and how much of it is left
#pragma unroll 1
  for (int guard = 0; guard < (1 << 26); guard++) {
    const bool part = __any_sync(FULL, ct > 0);
    const bool have = r0 < r1 || part || lm;
    const bool done = !have && m == 0;
    if (have) {
      int ti;
      bool pass;
      if (r0 < r1) {
        ti = r0 + lane;
        pass = ti < r1;
        r0 += 32;
      } else {
        if (!part) {
          const int l0 = __ffs(lm) - 1;
          lm &= lm - 1;
          const int l1 = lm ? __ffs(lm) - 1 : -1;
          lm &= lm - 1;
          const int src = lane < 16 ? l0 : l1;
          st = __shfl_sync(FULL, r.start, src & 31);
          ct = __shfl_sync(FULL, r.count, src & 31);
          if (src < 0) ct = 0;
        }
        ti = st + (lane & 15);
        pass = (lane & 15) < ct;
        st += 16;
        ct -= 16;
      }
      if (pass) {
        const float4 cf = tv.posf[ti];
        pass = pair_d2_lo(Q.qx, Q.qy, Q.qz, cf.x, cf.y, cf.z, Q.two_eps) < Q.thr;
      }
      const unsigned pm = __ballot_sync(FULL, pass);
      if (pass) w.queue[Q.qn + __popc(pm & ((1u << lane) - 1u))] = ti;
      Q.qn += __popc(pm);
    }
    if (Q.qn >= 32 || (done && Q.qn > 0)) {
      __syncwarp();
      const int cnt = min(32, Q.qn), rest = Q.qn - cnt;
      wq_flush<S>(Q, w, tv, lane, cnt);
      __syncwarp();
      const int moved = lane < rest ? w.queue[32 + lane] : 0;
      __syncwarp();
      if (lane < rest) w.queue[lane] = moved;
      Q.qn = rest;
    }
    if (done) return true;
    if (have) continue;
    // the next nodes
    bool need = false;
    if (lane < m) {
      r = tv.node[tv.nbase + h];
      need = box_d2_lo(Q.qx, Q.qy, Q.qz, Q.eps, r) < Q.thr;
    }
    const bool leaf = need && r.count <= tv.b;
    const unsigned inner = __ballot_sync(FULL, need && !leaf);
    lm = __ballot_sync(FULL, leaf);
    const int ne = __popc(inner);
    if (sp + 2 * ne > kWqStack) return false;
    if ((inner >> lane) & 1u) {  // the children of the lowest lane's node end on top
      const int slot = sp + 2 * __popc((inner >> lane) >> 1);
      w.stk[slot] = 2 * h + 2;
      w.stk[slot + 1] = 2 * h + 1;
    }
    sp += 2 * ne;
    __syncwarp();
    m = sp <= kWqBatchLimit ? min(32, sp) : 1;
    m = min(m, sp);
    if (lane < m) h = w.stk[sp - 1 - lane];
    sp -= m;
    __syncwarp();
  }
  return false;
}

// Heap index, first particle and size of the smallest node on the path of tree index
// `self` that holds at least `want` particles (the root if none is smaller).
__device__ __forceinline__ void wq_home(const TreeView& tv, int self, int want, int& h,
                                        int& start, int& size) {
  int i = self - tv.pstart;
  int hh = 0, s0 = 0, sz = tv.n;
  h = 0;
  start = tv.pstart;
  size = tv.n;
  while (sz > tv.b) {
    int ls = (sz - 1) / 2 + 1;  // KDTree.cxx:1012, 1025-1030
    if (i < s0 + ls) {
      hh = 2 * hh + 1;
      sz = ls;
    } else {
      hh = 2 * hh + 2;
      s0 += ls;
      sz -= ls;
    }
    if (sz < want) break;
    h = hh;
    start = tv.pstart + s0;
    size = sz;
  }
}

// The same for a query point that is no particle: the path follows the split planes
// (SplitNode's left child holds the coordinates up to the split value).
__device__ __forceinline__ void wq_home_point(const TreeView& tv, const double x[3], int want,
                                              int& h, int& start, int& size) {
  h = 0;
  start = tv.pstart;
  size = tv.n;
  while (size > tv.b) {
    const NodeX& nx = tv.nodex[tv.nbase + h];
    const int d = nx.split_dim;
    const double c = d == 0 ? x[0] : (d == 1 ? x[1] : x[2]);
    const int ch = 2 * h + (c > nx.split_val ? 2 : 1);
    const NodeRec& r = tv.node[tv.nbase + ch];
    if (r.count < want) break;
    h = ch;
    start = r.start;
    size = r.count;
  }
}

// An FP32 upper bound of the k-th distance from the query's own subtree [hs, hs + hn):
// a value T with at least K particles whose FP32 upper bound of the squared distance is
// at or below T (bisection over the bit patterns, which order as the non-negative values
// do), for a target search counting only particles provably at a non-zero distance and other
// than the query (it skips those). Returns +inf when fewer than K qualify. A subtree larger
// than 32 R particles (a large leaf) gives the bound of its first ones.
template <int S>
__device__ __forceinline__ float wq_home_bound(const WqQuery<S>& Q, const TreeView& tv, int lane,
                                               int self, int hs, int hn, int K,
                                               bool target) {
  const unsigned FULL = 0xffffffffu;
  constexpr int R = 2 * S + 1;
  unsigned hb[R];
  unsigned mn = 0x7f800000u, mx = 0u;
#pragma unroll
  for (int r = 0; r < R; r++) {
    int c = r * 32 + lane;
    hb[r] = 0x7f800000u;
    if (c < hn) {
      int ti = hs + c;
      float4 cf = tv.posf[ti];
      float lo = pair_d2_lo(Q.qx, Q.qy, Q.qz, cf.x, cf.y, cf.z, Q.two_eps);
      if (!target || (ti != self && lo > 0.f)) {
        hb[r] = __float_as_uint(pair_d2_hi(Q.qx, Q.qy, Q.qz, cf.x, cf.y, cf.z, Q.two_eps));
        mn = min(mn, hb[r]);
        mx = max(mx, hb[r]);
      }
    }
  }
  mn = __reduce_min_sync(FULL, mn);
  mx = __reduce_max_sync(FULL, mx);
  int cnt = 0;
#pragma unroll
  for (int r = 0; r < R; r++) cnt += hb[r] <= mx ? 1 : 0;
  if (__reduce_add_sync(FULL, cnt) < K) return __uint_as_float(0x7f800000u);
  // invariant: count(<= hi) >= K; 14 halvings bring hi within 2^-14 of the span
  unsigned lo = mn, hi = mx;
  for (int it = 0; it < 14 && lo < hi; it++) {
    unsigned mid = lo + ((hi - lo) >> 1);
    int c = 0;
#pragma unroll
    for (int r = 0; r < R; r++) c += hb[r] <= mid ? 1 : 0;
    if (__reduce_add_sync(FULL, c) >= K) hi = mid;
    else lo = mid + 1;
  }
  return __uint_as_float(hi + 1u);  // strictly above: candidates test lo < thr
}

// The search of one query (tree index `self`, or -1 for a point; position x0): the direct
// pass (seeded with the subtree around the query) and, on a periodic tree, the image passes with
// the reference's gates. exclude_self: the target search of the direct pass skips the
// query and zero distances (KDLeafNode.cxx:19-21). On return Q.L holds the K nearest.
template <int S>
__device__ void wq_search(WqQuery<S>& Q, WqSmem& w, const KnnArgs& a, const TreeView& tv,
                          int lane, int self, const double x0[3], int K, bool exclude_self) {
  wq_init<S>(Q.L, lane, K);
  Q.K = K;
  Q.topk = __double_as_longlong(kMaxValue);
  Q.thr = thresh_hi_bits(Q.topk);
  Q.qn = 0;
  Q.self = exclude_self ? self : -1;
  wq_set_point<S>(Q, tv, x0);
  int home, r0, rn;
  if (self >= 0) wq_home(tv, self, K + 1, home, r0, rn);
  else wq_home_point(tv, x0, K + 1, home, r0, rn);
  // the bound lets the rest of the tree be pruned at once
  Q.thr = fminf(Q.thr, wq_home_bound<S>(Q, tv, lane, self, r0, rn, K, exclude_self));
  int near_sq = 0, near_lin = 0;
  bool ok = true;
#pragma unroll 1
  for (int pass = 0; pass < 8 && ok; pass++) {
    // pass 0 searches around the query; the image passes follow in the reference's order
    if (pass > 0) {
      if (!a.periodic) break;
      const int mk = kImageMask[pass];
      const bool lin = !(pass <= 3 || a.min_image);
      if (pass == 1) {
        // the k-th distance only shrinks, so walls ruled out after the direct pass stay ruled out
        Q.self = -1;
        const float4 qf = make_float4(__double2float_rn(x0[0]), __double2float_rn(x0[1]),
                                      __double2float_rn(x0[2]), 0.f);
        const float top_hi = thresh_hi_bits(Q.topk);
        const float qeps = query_eps(tv, x0[0], x0[1], x0[2]);
        near_sq = near_walls(qf, tv.period, qeps, top_hi);
        near_lin = near_walls_lin(qf, tv.period, qeps, top_hi);
      }
      if ((mk & ~(lin ? near_lin : near_sq)) != 0) continue;
      double xq[3];
      const double sval = reflect(x0, xq, tv.period, mk);
      const double top = __longlong_as_double(Q.topk);
      // KDSplitNode.cxx:1129 gates 1-D images with sqrt(top) > sval, :1134-1146 the 2-D
      // and 3-D images with top > sval
      if (!(lin ? (top > sval) : (dsqrt_call(top) > sval))) continue;
      wq_set_point<S>(Q, tv, xq);
      home = -1;
      r0 = rn = 0;
    }
    ok = wq_pass<S>(Q, w, tv, lane, home, r0, r0 + rn);
  }
  if (!ok && lane == 0) atomicExch(a.err, kErrCapacity);
}

// Rank of each list entry among the first K by value (ties by position): the nsmooth
// smallest |dv| of CalcVelDensity are those of rank < nsmooth.
template <int S>
__device__ __forceinline__ void wq_ranks(const long long v[S], int lane, int K, int rank[S]) {
#pragma unroll
  for (int s = 0; s < S; s++) rank[s] = 0;
  for (int p = 0; p < K; p++) {
    long long vp = v[0];
#pragma unroll
    for (int s = 1; s < S; s++)
      if ((p >> 5) == s) vp = v[s];
    vp = __shfl_sync(0xffffffffu, vp, p & 31);
#pragma unroll
    for (int s = 0; s < S; s++) {
      int me = s * 32 + lane;
      rank[s] += (vp < v[s] || (vp == v[s] && p < me)) ? 1 : 0;
    }
  }
}

static __device__ __noinline__ double two_rsqrt_call(double t) { return 1.0 / (0.5 * __dsqrt_rn(t)); }
// 2 / sqrt(t) (the 1/h of h = sqrt(t) / 2) to about 2e-16 relative: the FP32 reciprocal
// square root as the start and two Newton steps y (3/2 - t/2 y^2) in FP64. Outside the
// FP32 normal range it takes the FP64 square root and division.
__device__ __forceinline__ double two_rsqrt(double t) {
  const float tf = __double2float_rn(t);
  if (!(tf > 1e-30f && tf < 1e30f)) return two_rsqrt_call(t);
  double y = (double)rsqrtf(tf);
  const double ht = 0.5 * t;
  y = dmul(y, __fma_rn(-ht, dmul(y, y), 1.5));
  y = dmul(y, __fma_rn(-ht, dmul(y, y), 1.5));
  return 2.0 * y;
}
// 1 / x to about 2e-16 relative: the FP32 reciprocal and two Newton steps y (2 - x y).
__device__ __forceinline__ double recip_newton(double x) {
  const float xf = __double2float_rn(x);
  if (!(xf > 1e-30f && xf < 1e30f)) return 1.0 / x;
  double y = (double)__frcp_rn(xf);
  y = dmul(y, __fma_rn(-x, y, 2.0));
  y = dmul(y, __fma_rn(-x, y, 2.0));
  return y;
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = dadd(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

constexpr int kWqWpb = 8;  // warps (queries) per block

// What one query's k-list (L, topk: the key at position K - 1) becomes: neighbour rows
// ascending in d2 (kEpiNN), or the SPH sums. `qi` indexes the per-query outputs and `self`
// is the query's tree index. All lanes of the warp call this together.
template <int S, int EPI>
__device__ __forceinline__ void wq_epilogue(const KnnArgs& a, const TreeView& tv, int lane, int qi,
                                            int self, int K, const WqList<S>& L, long long topk) {
  const unsigned FULL = 0xffffffffu;
  const int kr = a.kernres;
  const double inv_delta = 0.5 * (double)(kr - 1);  // 1 / table step, exact
  if (EPI == kEpiNN) {
    // rows ascending in d2; the popped largest (FindNearestPos on a periodic tree) or the
    // nearest (FindNearest on a periodic tree: k + 1 searched, k written) are left out
    // exactly as the heap version pops them
    int first = K - (a.drop_largest ? 1 : 0) - a.kout;
    size_t row = (size_t)qi * a.kout;
#pragma unroll
    for (int s = 0; s < S; s++) {
      int i = s * 32 + lane - first;
      if (i >= 0 && i < a.kout) {
        a.nn[row + i] = L.idx[s];
        a.d2[row + i] = __longlong_as_double(L.key[s]);
      }
    }
    return;
  }
  // density family: the list holds exactly the k neighbours (target search)
  bool missing = false;
#pragma unroll
  for (int s = 0; s < S; s++) missing |= (s * 32 + lane < K) && L.idx[s] < 0;
  if (__any_sync(FULL, missing)) {
    if (lane == 0) atomicExch(a.err, kErrTooFew);
    // no row: what reads the saved rows skips it
    if (EPI == kEpiSave && lane == 0) a.nn[(size_t)qi * K + K - 1] = -1;
    if (EPI == kEpiDensSave && lane == 0) a.nn[(size_t)(self - tv.pstart) * K + K - 1] = -1;
    return;
  }
  if (EPI == kEpiSave) {
#pragma unroll
    for (int s = 0; s < S; s++)
      if (s * 32 + lane < K) a.nn[(size_t)qi * K + s * 32 + lane] = L.idx[s];
    return;
  }
  const double* T = a.kernel;
  if (EPI == kEpiDensity || EPI == kEpiDensVel || EPI == kEpiDensPart || EPI == kEpiDensSave) {
    // KDCalcSmoothQuantities.cxx:260-286: one neighbour per lane. 1 / h with
    // h = sqrt(top) / 2 (the reference divides by h) within a few ulps, far inside the
    // 1e-12 density tolerance
    const double me_m = EPI == kEpiDensPart ? 0.0 : tv.pos[self].m;
    double ih = two_rsqrt(__longlong_as_double(topk));
    double norm = dmul(dmul(ih, ih), ih);  // 1 / h^3 (the reference takes pow(h, 3))
    double wnorm = EPI == kEpiDensPart ? norm : 0.5 * norm;
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < S; s++) {
      int p = s * 32 + lane;
      if (p >= K) continue;
      double d2 = __longlong_as_double(L.key[s]);
      int j = L.idx[s];
      // the farthest neighbour sits at q = 2 exactly in the reference's arithmetic (the
      // table's last entry); the product with 1/h could land an ulp below it
      double q = dmul(sqrt_newton(d2), ih);
      double wq = L.key[s] == topk ? T[kr - 1] : wsm_line(q, kr, inv_delta, T);
      double wij = dmul(wq, wnorm);
      acc = dadd(acc, dmul(wij, tv.pos[j].m));
      if (EPI != kEpiDensPart) {
        atomicAdd(&a.rho[j], dmul(wij, me_m));
        if (EPI == kEpiDensSave) a.nn[(size_t)(self - tv.pstart) * K + p] = j;
      }
    }
    acc = warp_sum(acc);
    if (lane == 0) {
      if (EPI == kEpiDensPart) a.rho[qi] = acc;
      else atomicAdd(&a.rho[self], acc);
    }
  }
  if (EPI == kEpiDensVel || EPI == kEpiVel || EPI == kEpiVelPart) {
    // KDCalcSmoothQuantities.cxx:354-383: |dv| of the Nsearch neighbours, keep the
    // Nsmooth smallest, h = 0.5 max, sum Wsm(|dv|/h) h^-3 with unit weights
    const V4 vi = self >= 0 ? tv.vel[self]
                            : make_v4(a.qv[3 * (size_t)qi], a.qv[3 * (size_t)qi + 1],
                                      a.qv[3 * (size_t)qi + 2], 0.0);
    long long vk[S];
#pragma unroll
    for (int s = 0; s < S; s++) {
      vk[s] = kWqSent;
      if (s * 32 + lane < K) {
        V4 vj = tv.vel[L.idx[s]];
        vk[s] = dkey(sqrt_newton(dist2_exact(vi.x, vi.y, vi.z, vj.x, vj.y, vj.z)));
      }
    }
    int ns = a.nsmooth;
    bool sel[S];
    if (ns < K) {
      int rk[S];
      wq_ranks<S>(vk, lane, K, rk);
#pragma unroll
      for (int s = 0; s < S; s++) sel[s] = s * 32 + lane < K && rk[s] < ns;
    } else {
#pragma unroll
      for (int s = 0; s < S; s++) sel[s] = s * 32 + lane < K;
    }
    long long vmaxk = 0;
#pragma unroll
    for (int s = 0; s < S; s++)
      if (sel[s]) vmaxk = max(vmaxk, vk[s]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmaxk = max(vmaxk, __shfl_xor_sync(FULL, vmaxk, o));
    double ih = recip_newton(0.5 * __longlong_as_double(vmaxk));
    double norm = dmul(dmul(ih, ih), ih);
    double acc = 0.0;
#pragma unroll
    for (int s = 0; s < S; s++) {
      if (!sel[s]) continue;
      double q = dmul(__longlong_as_double(vk[s]), ih);
      double wq = vk[s] == vmaxk ? T[kr - 1] : wsm_line(q, kr, inv_delta, T);  // q = 2
      acc = dadd(acc, dmul(wq, norm));
    }
    acc = warp_sum(acc);
    if (lane == 0) {
      if (EPI == kEpiVelPart) a.vden[qi] = acc;
      else a.vden[self] = acc;
    }
  }
}

// One query's search and epilogue on one warp (as wq_epilogue).
template <int S, int EPI>
__device__ void wq_run(const KnnArgs& a, const TreeView& tv, WqSmem& w, int lane, int qi,
                       int self, const double x0[3], int K) {
  WqQuery<S> Q;
  wq_search<S>(Q, w, a, tv, lane, self, x0, K, a.exclude_self != 0);
  wq_epilogue<S, EPI>(a, tv, lane, qi, self, K, Q.L, Q.topk);
}

}  // namespace
}  // namespace nbk
