// Phase-space nearest neighbours of every particle of a tree (FindNearest and CalcDensity on
// a TreeType TPHS tree without images, phase.cu names the reference's functions): a warp per
// group of neighbouring particles.
//
// What bounds it: with a lane per query (phase.cu, 32 queries a warp) every accepted
// candidate costs its lane an FP64 distance and a heap insertion while the others wait, about
// 130 a query, and the FP64 pipe (16 cycles a warp instruction, however few lanes are active)
// was 69% busy at 11 active lanes. Here a warp walks the tree once for a group of up to G
// particles, tests each opened leaf's particles 32 at a time for every query that wants the
// leaf, in FP32, and the K nearest are found by selection from buffers (knn_select.cuh); FP64
// distances are left for the neighbours themselves, a neighbour per lane.
//
// Both parts of the local-metric search run this way: the metric spacing
// (CalculateMetricSpacing: the 8 nearest in the plain distance) and the exact K nearest in the
// query's own metric. The reference prunes that search with unscaled offsets, so its answer
// is the exact one only where no particle of the exact K lies in a cell it prunes. A cell is
// pruned when its unscaled offset sum, which is at most the plain squared distance of any of
// its particles, reaches the heap top of the moment, which is never below the exact K-th
// metric distance. So the exact K are the reference's answer when every weight is at least
// 1 + 1e-9 (the plain distance is then below the metric one), and also whenever the largest
// plain squared distance among them is below their K-th metric one (by 1e-9); the few other
// queries are walked in the reference's order by a warp each (k_phase_walk).
//
// What FP32 cannot resolve -- a candidate not provably at a non-zero distance, more
// candidates than a buffer holds within the rounding of the K-th (a weight of 1e12, from an
// offset of 1e-6 to the second nearest, is enough) -- gets the exact K in FP64 from a block
// of its own (k_phase_exact): in such a metric a cell is a slab of the whole box, one lane
// visiting it took up to 90 ms. Queries without a metric spacing take the lane-per-query
// kernel.
//
// Measured (2^18 clustered particles, local metric, CalcDensity(32); it depends on the seed):
// 6.3-14.7 ms, a lane per query 31-50 ms; the FP64 pipe and instruction issue are each half
// busy at 20 warps per SM (28 warps: 12.6 against 11.5 ms, spills). Offsets formed in FP64
// from the exact coordinates cost 11.5 ms where the FP32 copies and residuals cost 9.5.
//
// Coordinates are screened as FP32 offsets from the group's middle particle, formed from the
// FP32 copies and their residuals, so that their rounding is relative to the group's extent:
// with s the FP32 sum and d the distance, |sqrt(s) - d| <= E + 2^-20 sqrt(s),
// E = sqrt(sum w (2^-22 extent + 2^-19 eps)^2), eps the FP32 rounding of a coordinate.
#include <algorithm>

#include "knn_select.cuh"
#include "phase_core.cuh"

namespace nbk {
namespace {

constexpr int kPgWpb = 4;     // warps (groups) per block
constexpr int kPgStack = 192;
// nodes tested per step (2^18 clustered particles, k = 32: 32 at once 29 ms, 16 13 ms: the
// frontier grows before the K-th distances have shrunk)
constexpr int kPgPop = 16;

// One query's row in shared memory.
struct __align__(16) PgQuery {
  float q[6];    // offset from the group's centre
  float w[6];    // weights, rounded down
  float thr;     // FP32 squared distances above it cannot be among the K nearest
  float pad;
  float a[6];    // FP32 coordinates (node tests)
};

template <int S>
struct PgSmem {
  unsigned bs[GrpCfg<S>::G][GrpCfg<S>::cap];
  int bi[GrpCfg<S>::G][GrpCfg<S>::cap];
  PgQuery q[GrpCfg<S>::G];
  int stk[kPgStack];
};

// The group and the pass: queries of `act` look for their K nearest; lane q keeps query q's
// buffer count and E.
struct PgPass {
  int gs, gn;      // first particle (tree index), particles
  float4 ph, pl, vh, vl;  // centre: FP32 copies and residuals
  int cnt;
  float two_e;
  unsigned act;
  bool skip_self;
};

// Offsets of particle ti from the group's centre.
__device__ __forceinline__ void pg_offsets(const TreeView& tv, const PgPass& P, int ti, float c[6]) {
  const float4 p = tv.posf[ti], pr = tv.posr[ti], v = tv.velf[ti], vr = tv.velr[ti];
  c[0] = (p.x - P.ph.x) + (pr.x - P.pl.x);
  c[1] = (p.y - P.ph.y) + (pr.y - P.pl.y);
  c[2] = (p.z - P.ph.z) + (pr.z - P.pl.z);
  c[3] = (v.x - P.vh.x) + (vr.x - P.vl.x);
  c[4] = (v.y - P.vh.y) + (vr.y - P.vl.y);
  c[5] = (v.z - P.vh.z) + (vr.z - P.vl.z);
}

// Screen one candidate per lane (mask: the queries that want it) for every query of `any`.
template <int S>
__device__ __forceinline__ void pg_screen(PgSmem<S>& w, const TreeView& tv, PgPass& P, int lane,
                                          int ti, unsigned mask, int K) {
  const unsigned FULL = 0xffffffffu;
  constexpr int cap = GrpCfg<S>::cap;
  float c[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (mask) pg_offsets(tv, P, ti, c);
#pragma unroll 1
  for (unsigned any = __reduce_or_sync(FULL, mask) & P.act; any; any &= any - 1) {
    const int i = __ffs(any) - 1;
    const PgQuery& Q = w.q[i];
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const float d = c[k] - Q.q[k];
      s = __fmaf_rn(__fmul_rn(Q.w[k], d), d, s);
    }
    float thr = Q.thr;
    bool pass = ((mask >> i) & 1u) && s <= thr && !(P.skip_self && ti == P.gs + i);
    unsigned pm = __ballot_sync(FULL, pass);
    if (!pm) continue;
    int cnt = __shfl_sync(FULL, P.cnt, i);
    if (cnt + __popc(pm) > cap) {
      const GrpCut t = grp_tighten<S>(w.bs[i], w.bi[i], lane, cnt, K, min(kGrpSlack, cap - 32 - K),
                                      __shfl_sync(FULL, P.two_e, i));
      thr = fminf(thr, t.thr);
      cnt = t.cnt;
      pass = pass && s <= thr;
      pm = __ballot_sync(FULL, pass);
      if (cnt + __popc(pm) > cap) thr = -1.f;  // too many within the rounding of the K-th
      if (lane == 0) w.q[i].thr = thr;
      __syncwarp();
      if (thr < 0.f) P.act &= ~(1u << i);
    }
    if (thr >= 0.f) {
      if (pass) {
        const int d = cnt + __popc(pm & ((1u << lane) - 1u));
        w.bs[i][d] = __float_as_uint(s);
        w.bi[i][d] = ti;
      }
      cnt += __popc(pm);
    }
    if (lane == i) P.cnt = cnt;
  }
}

// One pass of the active queries over the tree: home first (the smallest real node with
// enough particles around the group), then the siblings of home and of its ancestors and
// their subtrees. Queries that drop out of P.act take the second launch.
template <int S>
__device__ void pg_walk(PgSmem<S>& w, const TreeView& tv, PgPass& P, int lane, int hh, int lev,
                        int hs, int hn, int K) {
  const unsigned FULL = 0xffffffffu;
  const NodeS* N = tv.nodes6 + tv.nbase;
  const NodeF6* F = tv.nodef6 + tv.nbase;
  if (lane == 0)
    for (int i = 0; i < P.gn; i++) w.q[i].thr = FLT_MAX;
  P.cnt = 0;
  __syncwarp();
  // this lane's query of the node tests: its coordinates widened by their rounding, weights
  constexpr int G = GrpCfg<S>::G, kPer = 32 / G;
  float qlo[6], qhi[6], qw[6];
  {
    const PgQuery& Q = w.q[min(lane % G, P.gn - 1)];
#pragma unroll
    for (int k = 0; k < 6; k++) {
      qlo[k] = __fsub_rd(Q.a[k], tv.eps6[k]);
      qhi[k] = __fadd_ru(Q.a[k], tv.eps6[k]);
      qw[k] = Q.w[k];
    }
  }
  int sp = 0, m = 0, h = 0;
  int at = hs, end = hs + hn;  // the range or leaves being screened
  unsigned lm = 0;             // leaves of the last step not screened yet (a bit per lane)
  unsigned want = 0;           // the queries that want this lane's node
  int r_start = 0, r_count = 0, st = 0, ct = 0;
  unsigned mk = 0;
  bool home = true;
#pragma unroll 1
  for (int guard = 0; guard < (1 << 24); guard++) {
    if (home) {
      if (at < end) {
        pg_screen<S>(w, tv, P, lane, at + lane, at + lane < end ? P.act : 0u, K);
        at += 32;
        continue;
      }
      // the bounds from home, then the siblings, the nearest on lane 0
      home = false;
      __syncwarp();
#pragma unroll 1
      for (unsigned a = P.act; a; a &= a - 1) {
        const int i = __ffs(a) - 1;
        const int cnt = __shfl_sync(FULL, P.cnt, i);
        if (cnt < K) continue;
        const GrpCut t = grp_tighten<S>(w.bs[i], w.bi[i], lane, cnt, K, kGrpSlack,
                                        __shfl_sync(FULL, P.two_e, i));
        if (lane == 0) w.q[i].thr = t.thr;
        if (lane == i) P.cnt = t.cnt;
        if (t.thr < 0.f) P.act &= ~(1u << i);
      }
      __syncwarp();
      m = lev;
      if (lane < lev) {
        const int a = ((hh + 1) >> lane) - 1;
        h = (a & 1) ? a + 1 : a - 1;
      }
    }
    if (__any_sync(FULL, ct > 0) || lm) {
      // two leaves at a time, one per half warp, 16 particles a step
      if (!__any_sync(FULL, ct > 0)) {
        const int l0 = __ffs(lm) - 1;
        lm &= lm - 1;
        const int l1 = lm ? __ffs(lm) - 1 : -1;
        lm &= lm - 1;
        const int src = lane < 16 ? l0 : l1;
        st = __shfl_sync(FULL, r_start, src & 31);
        ct = __shfl_sync(FULL, r_count, src & 31);
        mk = __shfl_sync(FULL, want, src & 31);
        if (src < 0) ct = 0;
      }
      pg_screen<S>(w, tv, P, lane, st + (lane & 15), (lane & 15) < ct ? mk : 0u, K);
      st += 16;
      ct -= 16;
      continue;
    }
    if (m == 0 || !P.act) return;
    // the next nodes, 32 / G at a time: a lane per (node, query)
    want = 0;
    const bool mine = (P.act >> (lane % G)) & 1u;
    const float thr = w.q[lane % G].thr;
#pragma unroll 1
    for (int r = 0; r < m; r += kPer) {
      const int hr = __shfl_sync(FULL, h, (r + lane / G) & 31);
      bool in = false;
      if (mine && r + lane / G < m) {
        const NodeF6 b = F[hr];
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 6; k++) {
          const float g =
              fmaxf(0.f, fmaxf(__fsub_rd(b.lo[k], qhi[k]), __fsub_rd(qlo[k], b.hi[k])));
          s = __fadd_rd(s, __fmul_rd(__fmul_rd(qw[k], g), g));
        }
        in = s <= thr;
      }
      const unsigned bm = __ballot_sync(FULL, in);
      if (lane >= r && lane < r + kPer) want = (bm >> (G * (lane - r))) & ((1u << G) - 1u);
    }
    if (lane >= m) want = 0;
    bool leaf = false;
    if (want) {
      const NodeS nd = N[h];
      r_start = nd.start;
      r_count = nd.count;
      leaf = nd.split_dim < 0;
    }
    const unsigned inner = __ballot_sync(FULL, want && !leaf);
    lm = __ballot_sync(FULL, leaf);
    const int ne = __popc(inner);
    if (sp + 2 * ne > kPgStack) {
      P.act = 0;
      return;
    }
    if ((inner >> lane) & 1u) {
      const int slot = sp + 2 * __popc((inner >> lane) >> 1);
      w.stk[slot] = 2 * h + 2;
      w.stk[slot + 1] = 2 * h + 1;
    }
    sp += 2 * ne;
    __syncwarp();
    // near the stack's end one node at a time: a depth-first descent adds at most the depth
    m = sp <= kPgStack - 4 * kPgPop - 32 ? min(kPgPop, sp) : 1;
    m = min(m, sp);
    if (lane < m) h = w.stk[sp - 1 - lane];
    sp -= m;
    __syncwarp();
  }
  P.act = 0;
}

// The metric spacing of query i from its buffer of the 8 nearest (phase.cu
// ph_spacing_from_heap): the offsets to the second nearest, or to the next one whose offsets
// are all non-zero. Lane i gets them; false: the second launch.
template <int S>
__device__ __forceinline__ bool pg_spacing(PgSmem<S>& w, const TreeView& tv, PgPass& P, int lane,
                                           int i, double sr0[6], double& kvol) {
  const unsigned FULL = 0xffffffffu;
  const int cnt = __shfl_sync(FULL, P.cnt, i);
  if (cnt < 8) return false;
  const GrpCut f = grp_tighten<S>(w.bs[i], w.bi[i], lane, cnt, 8, 0,
                                  __shfl_sync(FULL, P.two_e, i));
  if (f.thr < 0.f || f.cnt > 32) return false;
  const P4 xp = tv.pos[P.gs + i];
  const V4 xv = tv.vel[P.gs + i];
  const double x[6] = {xp.x, xp.y, xp.z, xv.x, xv.y, xv.z};
  long long key = kWqSent;
  int j = P.gs + i;
  if (lane < f.cnt) {
    j = w.bi[i][lane];
    key = dkey(phase_d2(x, tv.pos[j], tv.vel[j]));
  }
  __syncwarp();
  warp_sort_asc(key, j, lane);
  const P4 p = tv.pos[j];
  const V4 v = tv.vel[j];
  const double y[6] = {p.x, p.y, p.z, v.x, v.y, v.z};
  double s[6], kv = 1.0;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    s[k] = fabs(dsub(y[k], x[k]));
    kv = dmul(kv, s[k]);
  }
  const unsigned nz = __ballot_sync(FULL, lane > 0 && lane < 8 && kv != 0.0);
  const int src = nz ? __ffs(nz) - 1 : 7;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const double t = __shfl_sync(FULL, s[k], src);
    if (lane == i) sr0[k] = t;
  }
  const double t = __shfl_sync(FULL, kv, src);
  if (lane == i) kvol = t;
  return true;
}

// A query left to a later launch: its tree index and metric.
struct PgLeft {
  double m[6];
  int self;
  int coop;  // every weight is at least 1 + 1e-9
};

// Lists of the later launches, head: [0] exact search in FP64, [1] walks, [2] a lane per query.
struct PgLists {
  int* head;
  PgLeft* exact;
  PgLeft* walk;
  int* redo;  // tree indices (without pstart)
  int max;    // entries of exact and of walk
};

// Append lane by lane where `mine`; a full list passes the query on to the lane-per-query one.
__device__ __forceinline__ void pg_leave(const PgLists& ls, int which, const TreeView& tv,
                                         const double m[6], int self, bool coop) {
  const int slot = atomicAdd(&ls.head[which], 1);
  if (slot < ls.max) {
    PgLeft x;
#pragma unroll
    for (int k = 0; k < 6; k++) x.m[k] = m[k];
    x.self = self;
    x.coop = coop;
    (which ? ls.walk : ls.exact)[slot] = x;
  } else {
    ls.redo[atomicAdd(&ls.head[2], 1)] = self - tv.pstart;
  }
}

// Whether the reference's pruning keeps the exact K nearest: their largest plain squared
// distance against the K-th metric one (bit patterns).
__device__ __forceinline__ bool pg_unpruned(long long u, long long top) {
  return dmul(__longlong_as_double(u), 1.0 + 1e-9) < __longlong_as_double(top);
}

template <int S, int EPI, bool METRIC>
__global__ void __launch_bounds__(32 * kPgWpb, 5) k_phase_group(PhaseArgs pa, PgLists ls,
                                                                int depth) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PgSmem<S>& w = reinterpret_cast<PgSmem<S>*>(smem_raw)[threadIdx.x >> 5];
  const unsigned FULL = 0xffffffffu;
  const KnnArgs& a = pa.k;
  const TreeView& tv = a.tv;
  const int lane = lane_id();
  const int g = blockIdx.x * kPgWpb + (threadIdx.x >> 5);
  if (g >= (1 << depth)) return;
  constexpr int G = GrpCfg<S>::G;
  const int K = a.kheap;
  // the group, and the smallest real node around it with more than K (and 8) particles (2 and 4
  // times as many were no faster)
  const int want = max(max(K + 1, G), 9);
  int s0 = 0, sz = tv.n, hh = 0, hs = 0, hn = tv.n, lev = 0;
  for (int i = depth - 1; i >= 0; i--) {
    const int ls0 = (sz - 1) / 2 + 1;
    const bool real = sz > tv.b;
    const int right = (g >> i) & 1;
    if (right) s0 += ls0;
    sz = right ? sz - ls0 : ls0;
    if (real && sz >= want) {
      hh = 2 * hh + 1 + right;
      hs = s0;
      hn = sz;
      lev++;
    }
  }
  PgPass P;
  P.gs = tv.pstart + s0;
  P.gn = sz;
  {
    const int mid = P.gs + (sz >> 1);
    P.ph = tv.posf[mid];
    P.pl = tv.posr[mid];
    P.vh = tv.velf[mid];
    P.vl = tv.velr[mid];
  }
  float far[6];
  {
    float o[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (lane < sz) {
      const float4 p = tv.posf[P.gs + lane], v = tv.velf[P.gs + lane];
      const float y[6] = {p.x, p.y, p.z, v.x, v.y, v.z};
      PgQuery& Q = w.q[lane];
      pg_offsets(tv, P, P.gs + lane, o);
#pragma unroll
      for (int k = 0; k < 6; k++) {
        Q.q[k] = o[k];
        Q.a[k] = y[k];
        Q.w[k] = 1.f;
      }
    }
#pragma unroll
    for (int k = 0; k < 6; k++)
      far[k] = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(fabsf(o[k]))));
  }
  __syncwarp();
  const unsigned all = (1u << sz) - 1u;
  // 2E of weights u: each offset carries 2^-23 of it (both ends) and its residual's rounding
  // (far below 2^-19 eps); the parts proportional to the distance are in the relative margin
  // of grp_thresh
  auto two_e_of = [&](const float u[6]) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const float e = __fadd_ru(__fmul_ru(far[k], 1.f / 4194304.f),
                                __fmul_ru(tv.eps6[k], 1.f / 524288.f));
      s = __fadd_ru(s, __fmul_ru(__fmul_ru(__fmul_ru(u[k], 1.0001f), e), e));
    }
    return __fmul_ru(__fsqrt_ru(s), 2.02f);
  };
  const float ones[6] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
  P.two_e = two_e_of(ones);
  unsigned okm = all, redo = 0u, coopm = all, walk = 0u, exact = 0u;
  double sr0[6] = {1, 1, 1, 1, 1, 1}, kvol = 1.0;
  double metric[6] = {1, 1, 1, 1, 1, 1};
  if (METRIC) {
    P.act = all;
    P.skip_self = false;
    pg_walk<S>(w, tv, P, lane, hh, lev, tv.pstart + hs, hn, 8);
    redo = all & ~P.act;
#pragma unroll 1
    for (unsigned left = P.act; left; left &= left - 1) {
      const int i = __ffs(left) - 1;
      if (!pg_spacing<S>(w, tv, P, lane, i, sr0, kvol)) redo |= 1u << i;
    }
    // a lane per query: the metric, and whether the exact search is the reference's
    bool coop = false, finite = false;
    if (lane < sz && !((redo >> lane) & 1u)) {
      double mmin = INFINITY, mmax = 0.0;
      float w32[6];
#pragma unroll
      for (int k = 0; k < 6; k++) {
        metric[k] = __ddiv_rn(1.0, dmul(sr0[k], sr0[k]));
        mmin = fmin(mmin, metric[k]);
        mmax = fmax(mmax, metric[k]);
        w32[k] = __double2float_rd(metric[k]);
        w.q[lane].w[k] = w32[k];
      }
      coop = mmin >= 1.0 + 1e-9;
      finite = mmax < 1e30;
      P.two_e = two_e_of(w32);
    }
    redo = __reduce_or_sync(FULL, redo);
    coopm = __ballot_sync(FULL, coop);
    okm = __ballot_sync(FULL, finite);
    walk = all & ~redo & ~okm;  // a zero offset: the walk's own handling of infinite weights
    __syncwarp();
  }
  // the search itself
  P.act = okm;
  P.skip_self = true;
  pg_walk<S>(w, tv, P, lane, hh, lev, tv.pstart + hs, hn, K);
  exact = okm & ~P.act;
  okm = P.act;
  long long top = 0;
#pragma unroll 1
  for (unsigned left = P.act; left; left &= left - 1) {
    const int i = __ffs(left) - 1;
    const int cnt = __shfl_sync(FULL, P.cnt, i), self = P.gs + i;
    const float e2 = __shfl_sync(FULL, P.two_e, i);
    bool ok = cnt >= K;
    GrpCut f{};
    if (ok) {
      f = grp_tighten<S>(w.bs[i], w.bi[i], lane, cnt, K, 0, e2);
      // every neighbour must be provably at a non-zero distance: sqrt(s) (1 - 2^-20) > E
      ok = f.thr >= 0.f && f.smin > __fmul_ru(__fmul_ru(e2, e2), 1.01f) && f.cnt <= 32 * S + 32;
    }
    if (!ok) {
      exact |= 1u << i;
      okm &= ~(1u << i);
      continue;
    }
    const P4 xp = tv.pos[self];
    const V4 xv = tv.vel[self];
    const double x[6] = {xp.x, xp.y, xp.z, xv.x, xv.y, xv.z};
    double m6[6];
    if (METRIC)
#pragma unroll
      for (int k = 0; k < 6; k++) m6[k] = __shfl_sync(FULL, metric[k], i);
    if (EPI == kPhNN || f.cnt > K) {
      long long key[S + 1];
      int idx[S + 1];
#pragma unroll
      for (int s = 0; s <= S; s++) {
        const int p = s * 32 + lane;
        key[s] = 0;
        idx[s] = -1;
        if (p < f.cnt) {
          idx[s] = w.bi[i][p];
          const P4 y = tv.pos[idx[s]];
          const V4 v = tv.vel[idx[s]];
          key[s] = dkey(METRIC ? metric_d2(x, y, v, m6) : phase_d2(x, y, v));
        }
      }
      if (f.cnt > K) grp_keep<S>(key, idx, w.bi[i], lane, f.cnt, K);
      if (EPI == kPhNN) {
        long long kk[S];
        int jj[S];
#pragma unroll
        for (int s = 0; s < S; s++) {
          kk[s] = kWqSent;
          jj[s] = -1;
          if (f.cnt == K) {
            if (s * 32 + lane < K) {
              kk[s] = key[s];
              jj[s] = idx[s];
            }
          } else if (s * 32 + lane < K) {
            jj[s] = w.bi[i][s * 32 + lane];
            const P4 y = tv.pos[jj[s]];
            const V4 v = tv.vel[jj[s]];
            kk[s] = dkey(METRIC ? metric_d2(x, y, v, m6) : phase_d2(x, y, v));
          }
        }
        if (METRIC && !((coopm >> i) & 1u)) {
          long long mx = 0, ux = 0;
#pragma unroll
          for (int s = 0; s < S; s++)
            if (s * 32 + lane < K) {
              mx = max(mx, kk[s]);
              ux = max(ux, dkey(phase_d2(x, tv.pos[jj[s]], tv.vel[jj[s]])));
            }
          if (!pg_unpruned(warp_max_key(ux), warp_max_key(mx))) {
            walk |= 1u << i;
            continue;
          }
        }
        grp_sort<S>(kk, jj, lane);
        const size_t row = (size_t)(self - tv.pstart) * a.kout;
#pragma unroll
        for (int s = 0; s < S; s++) {
          const int p = s * 32 + lane;
          if (p < K) {
            a.nn[row + p] = jj[s] - tv.pstart;
            a.d2[row + p] = __longlong_as_double(kk[s]);
          }
        }
        continue;
      }
    }
    // the density's row of squared distances (fused: nothing is decided by them)
    double* row = reinterpret_cast<double*>(w.bs[i]);
    double d2[S];
    long long mx = 0, ux = 0;
    const bool check = METRIC && !((coopm >> i) & 1u);
#pragma unroll
    for (int s = 0; s < S; s++) {
      const int p = s * 32 + lane;
      d2[s] = kGrpNone;
      if (p < K) {
        const int j = w.bi[i][p];
        const P4 y = tv.pos[j];
        const V4 v = tv.vel[j];
        if (check) ux = max(ux, dkey(phase_d2(x, y, v)));
        const double c6[6] = {y.x, y.y, y.z, v.x, v.y, v.z};
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < 6; k++) {
          const double d = dsub(x[k], c6[k]);
          t = __fma_rn(METRIC ? dmul(m6[k], d) : d, d, t);
        }
        d2[s] = t;
        mx = max(mx, dkey(t));
      }
    }
    mx = warp_max_key(mx);
    if (check && !pg_unpruned(warp_max_key(ux), mx)) {
      walk |= 1u << i;
      okm &= ~(1u << i);
      continue;
    }
    if (lane == i) top = mx;
#pragma unroll
    for (int s = 0; s < S; s++) row[s * 32 + lane] = dkey(d2[s]) == mx ? kGrpFar : d2[s];
    __syncwarp();
  }
  if (EPI == kPhDensity) {
    // a lane per query: h = 0.5 sqrt(top), norm = h^-6 times the product of sqrt(metric[j])
    // (KDCalcSmoothQuantities.cxx:251-270), which is 1 over the product of the offsets
    const int kr = a.kernres;
    double c1 = 0.0, wn = 0.0, wm = 0.0;
    if ((okm >> lane) & 1u) {
      const double ih = two_rsqrt(__longlong_as_double(top)), ih2 = dmul(ih, ih);
      c1 = dmul(ih, 0.5 * (double)(kr - 1));
      wn = dmul(dmul(ih2, ih2), ih2);
      if (METRIC) wn = __ddiv_rn(wn, kvol);
      wn = 0.5 * wn;
      wm = dmul(wn, tv.pos[P.gs + lane].m);
    }
    __syncwarp();
    grp_sums<S>(w.bs, w.bi, tv.pos, a.rho + (P.gs - tv.pstart), a.rho - tv.pstart, a.kernel, kr,
                lane, okm, K, c1, wn, wm);
  }
  if ((walk >> lane) & 1u) pg_leave(ls, 1, tv, metric, P.gs + lane, false);
  if ((exact >> lane) & 1u) pg_leave(ls, 0, tv, metric, P.gs + lane, (coopm >> lane) & 1u);
  if ((redo >> lane) & 1u) ls.redo[atomicAdd(&ls.head[2], 1)] = P.gs + lane - tv.pstart;
}

// What the K nearest of one query become, a neighbour per lane and slot of the list.
template <int S, int EPI>
__device__ __forceinline__ void pg_output(const PhaseArgs& pa, const TreeView& tv, int lane,
                                          int self, const double m[6], int K, const WqList<S>& L,
                                          long long topk) {
  const unsigned FULL = 0xffffffffu;
  const KnnArgs& a = pa.k;
  if (EPI == kPhNN) {
    const size_t row = (size_t)(self - tv.pstart) * a.kout;
#pragma unroll
    for (int s = 0; s < S; s++) {
      const int p = s * 32 + lane;
      if (p < K) {
        a.nn[row + p] = L.idx[s] >= 0 ? L.idx[s] - tv.pstart : -1;
        a.d2[row + p] = __longlong_as_double(L.key[s]);
      }
    }
    return;
  }
  bool missing = false;
#pragma unroll
  for (int s = 0; s < S; s++) missing |= s * 32 + lane < K && L.idx[s] < 0;
  if (__any_sync(FULL, missing)) {
    if (lane == 0) atomicExch(a.err, kErrTooFew);
    return;
  }
  const int kr = a.kernres;
  const double ih = two_rsqrt(__longlong_as_double(topk)), ih2 = dmul(ih, ih);
  const double c1 = dmul(ih, 0.5 * (double)(kr - 1));
  double norm = dmul(dmul(ih2, ih2), ih2);
  if (pa.metric) {
    double temp = 1.0;
#pragma unroll
    for (int k = 0; k < 6; k++) temp = dmul(temp, dsqrt_call(m[k]));
    norm = dmul(norm, temp);
  }
  norm = 0.5 * norm;
  const double wm = dmul(norm, tv.pos[self].m);
  double acc = 0.0;
#pragma unroll
  for (int s = 0; s < S; s++) {
    if (s * 32 + lane >= K) continue;
    const int j = L.idx[s];
    const double wq = grp_w(L.key[s] == topk ? kGrpFar : __longlong_as_double(L.key[s]), c1, kr,
                            a.kernel);
    atomicAdd(&a.rho[j - tv.pstart], dmul(wq, wm));
    acc = dadd(acc, dmul(wq, tv.pos[j].m));
  }
  acc = warp_sum(acc);
  if (lane == 0) atomicAdd(&a.rho[self - tv.pstart], dmul(acc, norm));
}

// ---- the exact K nearest in FP64, a block per query
// Every leaf's exact box is tested in FP64 (a leaf per lane) against the warp's K-th distance
// of the moment; the particles of those inside it are tested a lane each and enter the warp's
// list. The first warp merges the lists.
constexpr int kPxWarps = 8;
template <int S>
struct PxSmem {
  long long key[kPxWarps][32 * S];
  int idx[kPxWarps][32 * S];
};

template <int S, int EPI>
__global__ void __launch_bounds__(32 * kPxWarps) k_phase_exact(PhaseArgs pa, PgLists ls,
                                                               int leaf0, int nslots) {
  __shared__ PxSmem<S> sm;
  const unsigned FULL = 0xffffffffu;
  const KnnArgs& a = pa.k;
  const TreeView& tv = a.tv;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int count = min(ls.head[0], ls.max), K = a.kheap;
  const NodeS* N = tv.nodes6 + tv.nbase;
  const NodeB6* B = tv.nodeb6 + tv.nbase;
  for (int e = blockIdx.x; e < count; e += gridDim.x) {
    const PgLeft q = ls.exact[e];
    const P4 xp = tv.pos[q.self];
    const V4 xv = tv.vel[q.self];
    const double x[6] = {xp.x, xp.y, xp.z, xv.x, xv.y, xv.z};
    WqList<S> L;
    wq_init<S>(L, lane, K);
    long long topk = __double_as_longlong(kMaxValue);
    auto take = [&](long long dk, int j) {  // a candidate per lane
      for (unsigned acc = __ballot_sync(FULL, dk < topk); acc; acc &= acc - 1) {
        const int src = __ffs(acc) - 1;
        const long long k = __shfl_sync(FULL, dk, src);
        const int i = __shfl_sync(FULL, j, src);
        if (k < topk) {
          wq_insert<S>(L, lane, K, k, i);
          topk = wq_key_at<S>(L, K - 1);
        }
      }
    };
    for (int h0 = leaf0 + warp * 32; h0 < nslots; h0 += 32 * kPxWarps) {
      const int h = h0 + lane;
      NodeS nd{};
      bool in = false;
      if (h < nslots) {
        nd = N[h];
        in = nd.count > 0 && nd.split_dim < 0 &&
             dmul(box_lb6(x, q.m, B[h]), kLbShrink) < __longlong_as_double(topk);
      }
      for (unsigned lm = __ballot_sync(FULL, in); lm; lm &= lm - 1) {
        const int src = __ffs(lm) - 1;
        const int st = __shfl_sync(FULL, nd.start, src), ct = __shfl_sync(FULL, nd.count, src);
        for (int c0 = 0; c0 < ct; c0 += 32) {
          const int j = st + c0 + lane;
          long long dk = kWqSent;
          if (c0 + lane < ct && j != q.self) {
            dk = dkey(pa.metric ? metric_d2(x, tv.pos[j], tv.vel[j], q.m)
                                : phase_d2(x, tv.pos[j], tv.vel[j]));
            if (dk == 0) dk = kWqSent;  // distance 0 is skipped
          }
          take(dk, j);
        }
      }
    }
#pragma unroll
    for (int s = 0; s < S; s++) {
      sm.key[warp][s * 32 + lane] = L.key[s];
      sm.idx[warp][s * 32 + lane] = L.idx[s];
    }
    __syncthreads();
    if (warp == 0) {
      for (int o = 1; o < kPxWarps; o++)
        for (int s = 0; s < S; s++) {
          const int j = sm.idx[o][s * 32 + lane];
          take(j >= 0 ? sm.key[o][s * 32 + lane] : kWqSent, j);
        }
      bool walk = false;
      if (pa.metric && !q.coop) {
        long long u = 0;
#pragma unroll
        for (int s = 0; s < S; s++)
          if (s * 32 + lane < K && L.idx[s] >= 0)
            u = max(u, dkey(phase_d2(x, tv.pos[L.idx[s]], tv.vel[L.idx[s]])));
        walk = !pg_unpruned(warp_max_key(u), topk);
      }
      if (walk) {
        if (lane == 0) pg_leave(ls, 1, tv, q.m, q.self, false);
      } else {
        pg_output<S, EPI>(pa, tv, lane, q.self, q.m, K, L, topk);
      }
    }
    __syncthreads();
  }
}

// ---- the local-metric search in the reference's order, a warp per query
// The walk of phase.cu's ph_walk (which tells why skipped subtrees change nothing), made by
// all lanes together; a leaf's particles are tested a lane each (no pruning decision falls
// inside a leaf, so their order does not matter), the heap is the sorted list in registers.
struct PgWalkSmem {
  double rd_at[kPhDepth], old_at[kPhDepth];
};

template <int S, int EPI>
__global__ void __launch_bounds__(256) k_phase_walk(PhaseArgs pa, PgLists ls) {
  __shared__ PgWalkSmem sm[8];
  const unsigned FULL = 0xffffffffu;
  const KnnArgs& a = pa.k;
  const TreeView& tv = a.tv;
  const int lane = lane_id();
  PgWalkSmem& w = sm[threadIdx.x >> 5];
  const int count = min(ls.head[1], ls.max);
  const int K = a.kheap;
  const NodeS* N = tv.nodes6 + tv.nbase;
  const NodeF6* F = tv.nodef6 + tv.nbase;
  const NodeB6* B = tv.nodeb6 + tv.nbase;
  for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < count; i += gridDim.x * 8) {
    const int self = ls.walk[i].self;
    double m[6], x[6];
    {
      const P4 p = tv.pos[self];
      const V4 v = tv.vel[self];
      x[0] = p.x;
      x[1] = p.y;
      x[2] = p.z;
      x[3] = v.x;
      x[4] = v.y;
      x[5] = v.z;
    }
    float q32[6], w32[6], e32[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
      m[k] = ls.walk[i].m[k];
      q32[k] = __double2float_rn(x[k]);
      w32[k] = __double2float_rd(m[k]);
      e32[k] = fmaxf(tv.eps6[k], __fmul_ru(__double2float_ru(fabs(x[k])), 1.2e-7f));
    }
    // the FP32 bounds' own error, squared, in the metric: where it is not small against the
    // heap top, subtrees that they would open are tested in FP64 (a coordinate per lane)
    float e0 = 0.f;
#pragma unroll
    for (int k = 0; k < 6; k++) e0 += w32[k] * (2.f * e32[k]) * (2.f * e32[k]);
    double xl = x[0], ml = m[0];
#pragma unroll
    for (int k = 1; k < 6; k++)
      if (lane == k) {
        xl = x[k];
        ml = m[k];
      }
    auto outside = [&](int node, float t, long long tk) {
      if (box_lb6f(q32, w32, e32, F[node]) >= t) return true;
      if (!(e0 > 1e-4f * t)) return false;
      const NodeB6& b = B[node];
      double s = 0.0;
      if (lane < 6) {
        const double lo = b.lo[lane], hi = b.hi[lane];
        const double g = xl < lo ? __dsub_rd(lo, xl) : (xl > hi ? __dsub_rd(xl, hi) : 0.0);
        s = __dmul_rd(__dmul_rd(ml, g), g);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) s = __dadd_rd(s, __shfl_xor_sync(FULL, s, o));
      s = __shfl_sync(FULL, s, 0);
      return dmul(s, kLbShrink) >= __longlong_as_double(tk);
    };
    WqList<S> L;
    wq_init<S>(L, lane, K);
    long long topk = __double_as_longlong(kMaxValue);
    float thr = thresh_hi_bits(topk);
    double off[6] = {0, 0, 0, 0, 0, 0};
    int h = 0, depth = 0, prev = -1;
    bool down = true;
    __syncwarp();
    if (lane == 0) w.rd_at[0] = 0.0;
    __syncwarp();
#pragma unroll 1
    for (int guard = 0; guard < (1 << 28); guard++) {
      bool up = false;  // done with h: back to its parent
      if (down && outside(h, thr, topk)) {
        up = true;
      } else {
        const NodeS nd = N[h];
        if (down && nd.split_dim < 0) {
          for (int c0 = 0; c0 < nd.count; c0 += 32) {
            const int j = nd.start + c0 + lane;
            long long dk = kWqSent;
            if (c0 + lane < nd.count && j != self) {
              const float4 pf = tv.posf[j], vf = tv.velf[j];
              const float c[6] = {pf.x, pf.y, pf.z, vf.x, vf.y, vf.z};
              if (pair_lb6f(q32, c, w32, e32) < thr) {
                dk = dkey(metric_d2(x, tv.pos[j], tv.vel[j], m));
                if (dk == 0) dk = kWqSent;  // distance 0 is skipped
              }
            }
            for (unsigned acc = __ballot_sync(FULL, dk < topk); acc; acc &= acc - 1) {
              const int src = __ffs(acc) - 1;
              const long long k = __shfl_sync(FULL, dk, src);
              const int jj = __shfl_sync(FULL, j, src);
              if (k < topk) {
                wq_insert<S>(L, lane, K, k, jj);
                topk = wq_key_at<S>(L, K - 1);
              }
            }
            thr = thresh_hi_bits(topk);
          }
          up = true;
        } else {
          const int cd = nd.split_dim;
          const double xc = get6(x, cd);
          const bool left_first = okey(xc) < okey(nd.split_val);
          const int nearh = left_first ? 2 * h + 1 : 2 * h + 2;
          const int farh = left_first ? 2 * h + 2 : 2 * h + 1;
          if (down) {
            if (depth + 1 >= kPhDepth) {
              if (lane == 0) atomicExch(a.err, kErrCapacity);
              break;
            }
            if (lane == 0) w.rd_at[depth + 1] = w.rd_at[depth];
            __syncwarp();
            prev = h;
            h = nearh;
            depth++;
            continue;
          }
          up = true;
          if (prev == nearh && !outside(farh, thr, topk)) {
            const double new_off = dsub(xc, nd.split_val);
            const double old = get6(off, cd);
            const double rdf =
                dadd(w.rd_at[depth], dadd(dmul(-old, old), dmul(new_off, new_off)));
            if (rdf < __longlong_as_double(topk)) {
              __syncwarp();
              if (lane == 0) {
                w.old_at[depth] = old;
                w.rd_at[depth + 1] = rdf;
              }
              set6(off, cd, new_off);
              __syncwarp();
              prev = h;
              h = farh;
              depth++;
              down = true;
              up = false;
            }
          } else if (prev == farh) {
            set6(off, cd, w.old_at[depth]);  // back from the farther child
          }
        }
      }
      if (up) {
        if (h == 0) break;
        prev = h;
        h = (h - 1) >> 1;
        depth--;
        down = false;
      }
    }
    pg_output<S, EPI>(pa, tv, lane, self, m, K, L, topk);
  }
}

template <int S, int EPI>
int launch_pg(const PhaseArgs& pa, DevAlloc& alloc, cudaStream_t st) {
  const KnnArgs& a = pa.k;
  const int64_t n = a.tv.n;
  int nsm = 0, dev = 0;
  NBK_CUDA_TRY(cudaGetDevice(&dev));
  NBK_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  int depth = 0;
  while (((n - 1) >> depth) + 1 > GrpCfg<S>::G) depth++;
  while ((1 << depth) < 16 * nsm && ((n - 1) >> (depth + 1)) + 1 >= 2) depth++;
  PgLists ls{};
  ls.max = (int)(n / 8 + 1024);
  std::vector<DevPart> parts{{(void**)&ls.head, sizeof(int) * 3},
                             {(void**)&ls.exact, sizeof(PgLeft) * ls.max},
                             {(void**)&ls.walk, sizeof(PgLeft) * ls.max},
                             {(void**)&ls.redo, sizeof(int) * n}};
  NBK_TRY(alloc.get_block(parts));
  NBK_CUDA_TRY(cudaMemsetAsync(ls.head, 0, sizeof(int) * 3, st));
  const size_t sm = sizeof(PgSmem<S>) * kPgWpb;
  const unsigned blocks = ((1u << depth) + kPgWpb - 1) / kPgWpb;
  if (pa.metric) {
    NBK_TRY(ensure_dyn_smem((const void*)k_phase_group<S, EPI, true>, (int)sm));
    k_phase_group<S, EPI, true><<<blocks, 32 * kPgWpb, sm, st>>>(pa, ls, depth);
  } else {
    NBK_TRY(ensure_dyn_smem((const void*)k_phase_group<S, EPI, false>, (int)sm));
    k_phase_group<S, EPI, false><<<blocks, 32 * kPgWpb, sm, st>>>(pa, ls, depth);
  }
  note_launch();
  // the leaves are on the last two levels of the heap-indexed nodes
  const int64_t slots = heap_slots(n, a.tv.b);
  k_phase_exact<S, EPI><<<(unsigned)nsm, 32 * kPxWarps, 0, st>>>(pa, ls, (int)(slots / 4),
                                                                 (int)slots);
  note_launch();
  if (pa.metric) {
    k_phase_walk<S, EPI><<<(unsigned)(2 * nsm), 256, 0, st>>>(pa, ls);
    note_launch();
  }
  NBK_CUDA_TRY(cudaGetLastError());
  PhaseArgs rest = pa;
  rest.k.qmode = 2;
  rest.k.qidx = ls.redo;
  rest.count = ls.head + 2;
  return launch_phase_lanes(rest, st);
}

template <int EPI>
int launch_pg_e(const PhaseArgs& pa, DevAlloc& alloc, cudaStream_t st) {
  if (pa.k.kheap <= 32) return launch_pg<1, EPI>(pa, alloc, st);
  if (pa.k.kheap <= 64) return launch_pg<2, EPI>(pa, alloc, st);
  return launch_pg<4, EPI>(pa, alloc, st);
}

}  // namespace

// Every particle of a tree, no images; the screened squares must stay inside FP32. Queries in
// no order, part of a tree or with images take a lane each (phase.cu).
bool phase_group_serves(const PhaseArgs& pa) {
  const KnnArgs& a = pa.k;
  if (pa.epi == kPhDensPart || a.qmode != 0 || a.q0 != 0 || a.nq != a.tv.n || a.periodic ||
      (pa.metric && pa.spacing_periodic) || a.kheap > 128 || a.kout != a.kheap ||
      a.nq < 4 * (std::max(a.kheap, 8) + 1))
    return false;
  for (int k = 0; k < 6; k++)
    if (!(a.tv.eps6[k] < 1e11f)) return false;
  return true;
}

int launch_phase_group(const PhaseArgs& pa, DevAlloc& alloc, cudaStream_t st) {
  if (pa.epi == kPhNN) return launch_pg_e<kPhNN>(pa, alloc, st);
  return launch_pg_e<kPhDensity>(pa, alloc, st);
}

}  // namespace nbk
