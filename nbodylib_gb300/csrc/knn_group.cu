// k-nearest-neighbour search of every particle of a tree, a compact group of particles per
// warp: the kNN behind CalcDensity, CalcVelDensity and FindNearest of all particles
// (KDTree::FindNearest(Int_t**, ...) and the loops of KDCalcSmoothQuantities.cxx:203-389).
//
// What bounds it, and why groups: with a warp per query (knn_wq.cuh) every query walks the
// tree alone, about 4,200 warp instructions a query at k = 32, most of them traversal and
// the sorted insertion of candidates that do not survive. Particles next to one another in
// tree order have nearly the same neighbourhood, so here one warp walks the tree once for a
// group of up to G particles, with a radius guessed from the density of the smallest node
// around the group with more than K particles, stages the particles within that radius of
// the group's box in shared memory, and every query only screens the staged ones, 32 lanes
// wide, keeping those within the radius in a buffer of its own. The K nearest are then found
// by selection (bisection over the FP32 squared distances), not by sorted insertion.
//
// Precision of the screen: a particle's coordinates are staged relative to the group's
// middle particle, as (hi - hi_c) + (lo - lo_c) from the FP32 copy posf (hi) and its FP32
// residual posr (lo). The error of a difference of two such offsets is bounded by a few
// 2^-23 of the offsets themselves (not of the coordinates), so the FP32 squared distance s
// and the true distance d satisfy |sqrt(s) - d| <= E + 2^-20 sqrt(s) with E of the order
// of 1e-6 of the group's extent, and the selection leaves the K nearest and hardly ever
// anything else; where it leaves more, FP64 distances (the reference's association
// ((dx*dx + dy*dy) + dz*dz)) decide.
//
// A query that this cannot answer exactly -- fewer than K particles within the radius, a
// candidate not provably at a non-zero distance (the target search skips zero distances,
// KDLeafNode.cxx:19-21), more candidates than the buffer holds within the rounding of the
// K-th, distances outside the FP32 range or not surely below the reference's MAXVALUE, a
// periodic query too close to an image gate -- and every query of a group whose box meets too
// many particles is appended to a list that a second launch serves with the warp-per-query
// search.
//
// The FP64 pipe (two operations per SM clock: 16 cycles a warp instruction) is the bound of
// the density sums. Per neighbour 13 FP64 instructions are left: 6 for the distance (fused;
// nothing is decided by it), 3 for the square root, 1 each for the table coordinate, the
// table line, the gathered and the scattered term. What belongs to a query and not to a
// neighbour (1/h, h^-3, products with the mass) is computed for all queries of the group at
// once, a lane per query, and the gathered terms are summed through shared memory, so these
// cost a group what they would cost one query.
//
// Measured (2^20 clustered particles, one GB300; the warp-per-query form in brackets):
// CalcDensity(32) 3.1 ms (6.0), 32768 uniform 0.098 ms (0.178), 256^3 with k = 64 70 + 69 ms
// (166 + 176). Groups of 16 took 4.0 ms (18 instead of 32 warps per SM), radii of 1.2 and
// 1.3 as the first 3.3; everything inlined 5.7 ms (instruction cache); first-pass failures
// and mixed groups left to the second launch 4.6 ms.
#include <algorithm>

#include "knn_select.cuh"

namespace nbk {
namespace {

constexpr int kGrpChunk = 64;   // candidates staged before the queries screen them
constexpr int kGrpStack = 192;  // frontier stack (node indices) per warp
constexpr int kGrpWpb = 4;      // warps (groups) per block
constexpr int kGrpStrict = 256;    // a group that stages more tests nodes query by query
constexpr int kGrpStaged = 1024;   // and one that stages more takes the second launch (12288:
                                   // 2^20 particles with a group that stages that many 5.4 ms, else 3.0;
                                   // 1024: 3.3 and 3.2)
// search radius of each pass in units of the expected K-th distance: a pass serves the
// queries that the one before found fewer than K particles for
constexpr int kGrpPasses = 3;
__device__ __constant__ static const float kGrpRadius[kGrpPasses] = {1.25f, 2.0f, 3.0f};

template <int S>
struct GrpSmem {
  float4 ch[kGrpChunk + 32];  // staged candidates: offsets from the centre, tree index
  // per query its candidates: FP32 squared distance and tree index; in the SPH sums the
  // row of bs holds 32 S doubles instead
  unsigned bs[GrpCfg<S>::G][GrpCfg<S>::cap];
  int bi[GrpCfg<S>::G][GrpCfg<S>::cap];
  float4 qs[GrpCfg<S>::G];  // the queries: offset from the centre, acceptance bound
  int stk[kGrpStack];
};

// The per-lane state of the group's queries (lane q < gn holds query q).
struct GrpLane {
  float x, y, z;  // offset from the centre
  float thr;      // FP32 squared distances above it are not taken; -1: the query takes the
                  // second launch
  int cnt;        // candidates in its buffer
  bool act;       // served by this pass
};

// Order-preserving map of floats to signed integers, and its inverse (the same map).
__device__ __forceinline__ int ford(float x) {
  const int i = __float_as_int(x);
  return i ^ ((i >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float ford_inv(int i) {
  return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}

// FP32 squared length, every use rounded the same way (explicit fused steps).
__device__ __forceinline__ float sq3(float x, float y, float z) {
  return __fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x)));
}

// Every live query screens the staged candidates [0, m).
template <int S>
__device__ __forceinline__ void grp_stream(GrpSmem<S>& w, GrpLane& L, int lane, int gs, int m, int K,
                           float two_e) {
  const unsigned FULL = 0xffffffffu;
  constexpr int cap = GrpCfg<S>::cap;
  // queries whose bound does not reach the box around the staged candidates skip them
  float blo[3], bhi[3];
  {
    int mn[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff};
    int mx[3] = {(int)0x80000000, (int)0x80000000, (int)0x80000000};
    for (int c0 = 0; c0 < m; c0 += 32) {
      if (c0 + lane >= m) continue;
      const float4 c = w.ch[c0 + lane];
      const int v[3] = {ford(c.x), ford(c.y), ford(c.z)};
#pragma unroll
      for (int d = 0; d < 3; d++) {
        mn[d] = min(mn[d], v[d]);
        mx[d] = max(mx[d], v[d]);
      }
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
      blo[d] = ford_inv(__reduce_min_sync(FULL, mn[d]));
      bhi[d] = ford_inv(__reduce_max_sync(FULL, mx[d]));
    }
  }
  const float gx = fmaxf(0.f, fmaxf(blo[0] - L.x, L.x - bhi[0]));
  const float gy = fmaxf(0.f, fmaxf(blo[1] - L.y, L.y - bhi[1]));
  const float gz = fmaxf(0.f, fmaxf(blo[2] - L.z, L.z - bhi[2]));
  // the screen's own distance of any of them is at least this (the same roundings, monotone)
  unsigned live = __ballot_sync(FULL, L.act && sq3(gx, gy, gz) <= L.thr);
  while (live) {
    const int q = __ffs(live) - 1;
    live &= live - 1;
    const float4 qs = w.qs[q];
    float thr = qs.w;
    int cnt = __shfl_sync(FULL, L.cnt, q);
#pragma unroll 1
    for (int c0 = 0; c0 < m; c0 += 32) {
      const float4 c = w.ch[c0 + lane];
      const int id = __float_as_int(c.w);
      const float s = sq3(c.x - qs.x, c.y - qs.y, c.z - qs.z);
      bool pass = c0 + lane < m && s <= thr && id != gs + q;
      unsigned pm = __ballot_sync(FULL, pass);
      if (!pm) continue;
      if (cnt + __popc(pm) > cap) {
        const GrpCut t = grp_tighten<S>(w.bs[q], w.bi[q], lane, cnt, K,
                                        min(kGrpSlack, cap - 32 - K), two_e);
        thr = fminf(thr, t.thr);
        cnt = t.cnt;
        pass = pass && s <= thr;
        pm = __ballot_sync(FULL, pass);
        if (cnt + __popc(pm) > cap) thr = -1.f;  // too many within the rounding of the K-th
        if (lane == q) L.thr = thr;
        if (lane == 0) w.qs[q].w = thr;
        if (thr < 0.f) break;
      }
      if (pass) {
        const int d = cnt + __popc(pm & ((1u << lane) - 1u));
        w.bs[q][d] = __float_as_uint(s);
        w.bi[q][d] = id;
      }
      cnt += __popc(pm);
    }
    if (lane == q) L.cnt = cnt;
  }
  __syncwarp();
}

// One group's constants.
struct GrpGeom {
  float qlo[3], qhi[3];  // box around the group's particles (FP32, widened)
  float4 ch, cl;         // the centre particle: FP32 copy and residual
  float reach;           // squared: particles farther from the box are of no use
};

__device__ __forceinline__ bool grp_near(const GrpGeom& ge, float lx, float ly, float lz, float hx,
                                         float hy, float hz) {
  const float gx = fmaxf(0.f, fmaxf(__fsub_rd(lx, ge.qhi[0]), __fsub_rd(ge.qlo[0], hx)));
  const float gy = fmaxf(0.f, fmaxf(__fsub_rd(ly, ge.qhi[1]), __fsub_rd(ge.qlo[1], hy)));
  const float gz = fmaxf(0.f, fmaxf(__fsub_rd(lz, ge.qhi[2]), __fsub_rd(ge.qlo[2], hz)));
  return __fadd_rd(__fadd_rd(__fmul_rd(gx, gx), __fmul_rd(gy, gy)), __fmul_rd(gz, gz)) <= ge.reach;
}

// Append the particle ti (one per lane, valid lanes only) to the staged candidates when it
// is within reach of the group's box. Its index carries the image pass (tag) it was found in.
template <int S>
__device__ __forceinline__ void grp_stage(GrpSmem<S>& w, const TreeView& tv, const GrpGeom& ge,
                                          int lane, bool valid, int ti, int tag, int& chn) {
  float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
  bool in = false;
  if (valid) {
    c = tv.posf[ti];
    in = grp_near(ge, c.x, c.y, c.z, c.x, c.y, c.z);
  }
  const unsigned pm = __ballot_sync(0xffffffffu, in);
  if (in) {
    const float4 r = tv.posr[ti];
    w.ch[chn + __popc(pm & ((1u << lane) - 1u))] =
        make_float4((c.x - ge.ch.x) + (r.x - ge.cl.x), (c.y - ge.ch.y) + (r.y - ge.cl.y),
                    (c.z - ge.ch.z) + (r.z - ge.cl.z), __int_as_float(ti | tag));
  }
  chn += __popc(pm);
}

// The nodes of one step tested query by query (a node per lane, `have` marks the lanes that
// hold one): whether any active query's bound reaches the lane's node. A node of more than K
// particles also bounds the K-th distance by its farthest corner, so a dense place inside a
// large radius cuts the bound before its particles are staged. Gaps are narrowed, and
// reaches widened, by the rounding of the offsets.
template <int S>
__device__ __forceinline__ bool grp_wanted(GrpSmem<S>& w, const GrpGeom& ge, GrpLane& L,
                                           const NodeRec& r, bool have, unsigned act, int lane,
                                           int K, float two_e) {
  const float lx = (r.lo[0] - ge.ch.x) - ge.cl.x, hx = (r.hi[0] - ge.ch.x) - ge.cl.x;
  const float ly = (r.lo[1] - ge.ch.y) - ge.cl.y, hy = (r.hi[1] - ge.ch.y) - ge.cl.y;
  const float lz = (r.lo[2] - ge.ch.z) - ge.cl.z, hz = (r.hi[2] - ge.ch.z) - ge.cl.z;
  const bool many = have && r.count > K;
  bool any = false;
#pragma unroll 1
  for (; act; act &= act - 1) {
    const int i = __ffs(act) - 1;
    float4 q = w.qs[i];
    const float ax = lx - q.x, bx = q.x - hx, ay = ly - q.y, by = q.y - hy, az = lz - q.z,
                bz = q.z - hz;
    // the farthest corner is at max(|lo - q|, |q - hi|) per dimension
    const float f = many ? sq3(fmaxf(fabsf(ax), fabsf(bx)), fmaxf(fabsf(ay), fabsf(by)),
                               fmaxf(fabsf(az), fabsf(bz)))
                         : FLT_MAX;
    const float fm = __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(f)));
    if (fm < q.w) {
      // widened twice: the bound of a cut to K of these candidates stays within it
      q.w = fminf(q.w, grp_thresh(grp_thresh(grp_thresh(fm, two_e), two_e), two_e));
      if (lane == i) {
        L.thr = q.w;
        w.qs[i].w = q.w;
      }
    }
    const float gx = fmaxf(0.f, fmaxf(ax, bx) - two_e);
    const float gy = fmaxf(0.f, fmaxf(ay, by) - two_e);
    const float gz = fmaxf(0.f, fmaxf(az, bz) - two_e);
    any = any || sq3(gx, gy, gz) <= q.w * (1.0f + 1.0f / 65536.0f);
  }
  __syncwarp();
  return have && any;
}

// Distance within which a box of extents e (sorted or not) with n particles is expected to
// hold K of them, taken as the largest of the line, square and cube estimates (the cube's
// unless the box is flat or thin). From logarithms: products of extents leave FP32's range
// where the extents are far inside it.
__device__ __forceinline__ float grp_radius(float ex, float ey, float ez, int n, int K) {
  const float a = fmaxf(ex, fmaxf(ey, ez)), c = fminf(ex, fminf(ey, ez));
  const float b = fmaxf(fminf(ex, ey), fminf(fmaxf(ex, ey), ez));
  const float f = __log2f(__fdividef((float)K, (float)n));
  const float la = __log2f(a), lb = __log2f(b), lc = __log2f(c);  // -inf where flat
  const float r1 = f + la - 1.f;
  const float r2 = (f + la + lb - 1.6515f) * 0.5f;                    // 1 / pi
  const float r3 = (f + la + lb + lc - 2.0665f) * (1.0f / 3.0f);     // 3 / (4 pi)
  return exp2f(fmaxf(r1, fmaxf(r2, r3)));
}

// One walk of the tree for the active queries: first home itself and the siblings of home
// and of its ancestors, one per lane (at most 31 levels), then their subtrees, up to 32
// nodes a step. Returns false when the queries have to take the second launch.
template <int S>
__device__ bool grp_walk(GrpSmem<S>& w, const TreeView& tv, GrpGeom& ge, GrpLane& L, int lane,
                         int gs, int hh, int lev, int tag, int K, float two_e) {
  const unsigned FULL = 0xffffffffu;
  const unsigned act = __ballot_sync(FULL, L.act);
  int chn = 0, nst = 0, sp = 0, m = lev + 1, h = hh;
  if (lane > 0 && lane <= lev) {
    const int a = ((hh + 1) >> (lane - 1)) - 1;
    h = (a & 1) ? a + 1 : a - 1;
  }
  unsigned lm = 0;      // leaves of the last step not staged yet (a bit per lane)
  NodeRec r{};
  int st = 0, ct = 0;   // the leaf this half warp stages, and how much of it is left
#pragma unroll 1
  for (int guard = 0; guard < (1 << 24); guard++) {
    const bool part = __any_sync(FULL, ct > 0);
    const bool done = m == 0 && lm == 0 && !part;
    // the queries screen the staged candidates when a further batch might not fit
    if (chn > kGrpChunk || (done && chn > 0)) {
      __syncwarp();
      grp_stream<S>(w, L, lane, gs, chn, K, two_e);
      nst += chn;
      chn = 0;
      // the bounds shrink as buffers are cut
      const float far = __uint_as_float(
          __reduce_max_sync(FULL, L.act && L.thr >= 0.f ? __float_as_uint(L.thr) : 0u));
      ge.reach = fminf(ge.reach, grp_thresh(far, two_e));
    }
    if (done) return true;
    if (part || lm) {
      // two leaves at a time, one per half warp, 16 particles a step
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
      grp_stage<S>(w, tv, ge, lane, (lane & 15) < ct, st + (lane & 15), tag, chn);
      st += 16;
      ct -= 16;
      continue;
    }
    // the next nodes
    bool need = false;
    if (lane < m) {
      r = tv.node[tv.nbase + h];
      need = grp_near(ge, r.lo[0], r.lo[1], r.lo[2], r.hi[0], r.hi[1], r.hi[2]);
    }
    // a group whose box meets a much denser place: nodes are tested query by query, so that
    // its cost stays that of its queries
    if (nst > kGrpStrict) need = grp_wanted<S>(w, ge, L, r, need, act, lane, K, two_e);
    const bool leaf = need && r.count <= tv.b;
    const unsigned inner = __ballot_sync(FULL, need && !leaf);
    lm = __ballot_sync(FULL, leaf);
    const int ne = __popc(inner);
    if (sp + 2 * ne > kGrpStack || nst > kGrpStaged) return false;
    if ((inner >> lane) & 1u) {
      const int slot = sp + 2 * __popc((inner >> lane) >> 1);
      w.stk[slot] = 2 * h + 2;
      w.stk[slot + 1] = 2 * h + 1;
    }
    sp += 2 * ne;
    __syncwarp();
    // above kWqBatchLimit entries pop one node at a time: a depth-first descent from there
    // adds at most the tree depth
    m = sp <= kWqBatchLimit ? min(32, sp) : 1;
    if (lane < m) h = w.stk[sp - 1 - lane];
    sp -= m;
    __syncwarp();
  }
  return false;
}

// The box around the active lanes' points, widened by e2.
template <int S>
__device__ __forceinline__ void grp_box(GrpGeom& ge, bool act, float4 p, float e2) {
  const unsigned FULL = 0xffffffffu;
  float lo[3], hi[3];
  lo[0] = act ? __fsub_rd(p.x, e2) : FLT_MAX;
  lo[1] = act ? __fsub_rd(p.y, e2) : FLT_MAX;
  lo[2] = act ? __fsub_rd(p.z, e2) : FLT_MAX;
  hi[0] = act ? __fadd_ru(p.x, e2) : -FLT_MAX;
  hi[1] = act ? __fadd_ru(p.y, e2) : -FLT_MAX;
  hi[2] = act ? __fadd_ru(p.z, e2) : -FLT_MAX;
#pragma unroll
  for (int d = 0; d < 3; d++) {
#pragma unroll
    for (int o = GrpCfg<S>::G / 2; o > 0; o >>= 1) {
      lo[d] = fminf(lo[d], __shfl_xor_sync(FULL, lo[d], o));
      hi[d] = fmaxf(hi[d], __shfl_xor_sync(FULL, hi[d], o));
    }
    ge.qlo[d] = __shfl_sync(FULL, lo[d], 0);
    ge.qhi[d] = __shfl_sync(FULL, hi[d], 0);
  }
}

// One group: on return lane q < gn holds the state of query gs + q and its buffer holds
// every particle whose FP32 squared distance is within thr.
template <int S>
__device__ void grp_search(GrpSmem<S>& w, const TreeView& tv, int lane, int g, int depth, int K,
                           GrpLane& L, int& gs, int& gn, float& two_e) {
  const unsigned FULL = 0xffffffffu;
  constexpr int G = GrpCfg<S>::G;
  // the group (the node at `depth` of the split rule, virtual below the leaves) and the
  // smallest real node around it with more than K particles (home)
  const int want = max(K + 1, G);
  int s0 = 0, sz = tv.n;
  int hh = 0, hn = tv.n, lev = 0;
  for (int i = depth - 1; i >= 0; i--) {
    const int ls = (sz - 1) / 2 + 1;  // KDTree.cxx:1012, 1025-1030
    const bool real = sz > tv.b;
    const int right = (g >> i) & 1;
    if (right) s0 += ls;
    sz = right ? sz - ls : ls;
    if (real && sz >= want) {
      hh = 2 * hh + 1 + right;
      hn = sz;
      lev++;
    }
  }
  gs = tv.pstart + s0;
  gn = sz;
  GrpGeom ge;
  ge.ch = tv.posf[gs + (gn >> 1)];
  ge.cl = tv.posr[gs + (gn >> 1)];
  const NodeRec home = tv.node[tv.nbase + hh];
  // a tree that fits the buffers is taken whole
  const float rad = tv.n <= GrpCfg<S>::cap
                        ? 1e18f
                        : grp_radius(__fsub_ru(home.hi[0], home.lo[0]),
                                     __fsub_ru(home.hi[1], home.lo[1]),
                                     __fsub_ru(home.hi[2], home.lo[2]), hn, K);
  // offsets of the queries from the group's middle particle
  float4 mine = make_float4(0.f, 0.f, 0.f, 0.f);
  L.thr = -1.f;
  L.cnt = 0;
  L.x = L.y = L.z = 0.f;
  if (lane < gn) {
    mine = tv.posf[gs + lane];
    const float4 r = tv.posr[gs + lane];
    L.x = (mine.x - ge.ch.x) + (r.x - ge.cl.x);
    L.y = (mine.y - ge.ch.y) + (r.y - ge.cl.y);
    L.z = (mine.z - ge.ch.z) + (r.z - ge.cl.z);
  }
  // 2E: an offset's error is at most 2^-23 of it plus the residuals' own rounding (2^-48 of
  // the coordinates, far below 2^-20 eps); the parts proportional to the distance are in
  // the relative margin of grp_thresh
  const float far = __uint_as_float(__reduce_max_sync(
      FULL, __float_as_uint(fmaxf(fabsf(L.x), fmaxf(fabsf(L.y), fabsf(L.z))))));
  two_e = __fmul_ru(4.f, __fadd_ru(__fmul_ru(far, 1.f / 4194304.f),
                                   __fmul_ru(tv.eps, 1.f / 524288.f)));
  const float e2 = __fmul_ru(2.f, tv.eps);  // the queries' own rounding and the candidates'
#pragma unroll 1
  for (int pass = 0; pass < kGrpPasses; pass++) {
    L.act = lane < gn && L.cnt < K;
    if (!__any_sync(FULL, L.act)) break;
    const float r = kGrpRadius[pass] * rad;
    grp_box<S>(ge, L.act, mine, e2);
    ge.reach = grp_thresh(r * r, two_e);
    if (L.act) {
      L.cnt = 0;
      L.thr = fminf(r * r, FLT_MAX);
      w.qs[lane] = make_float4(L.x, L.y, L.z, L.thr);
    }
    __syncwarp();
    if (!grp_walk<S>(w, tv, ge, L, lane, gs, hh, lev, 0, K, two_e)) {
      if (L.act) L.thr = -1.f;
      break;
    }
    if (L.act && L.thr < 0.f) L.cnt = K;  // given up: not tried again
  }
}

// Exact choice among the cnt > K candidates left in a query's buffer (at most 32 S + 32):
// FP64 distances, the largest dropped until K are left, their indices back in the buffer.
template <int S>
__device__ __noinline__ void grp_drop(int* bi, const P4* pos, int lane, int self, int cnt, int K) {
  const P4 x = pos[self];
  long long key[S + 1];
  int idx[S + 1];
#pragma unroll
  for (int s = 0; s <= S; s++) {
    const int p = s * 32 + lane;
    key[s] = 0;
    idx[s] = -1;
    if (p < cnt) {
      idx[s] = bi[p];
      const P4 c = pos[idx[s]];
      key[s] = dkey(dist2_exact(x.x, x.y, x.z, c.x, c.y, c.z));
    }
  }
  grp_keep<S>(key, idx, bi, lane, cnt, K);
}

// The neighbours of one query: its buffer cut to the K nearest (indices in bi[0 .. K)).
// Returns 0 when the query has to take the second launch, 2 when FP64 distances chose (the
// buffer's squared distances are then no longer those of its indices), else 1; thr returns an
// FP32 bound at or above the K-th squared distance.
template <int S>
__device__ int grp_select(GrpSmem<S>& w, const TreeView& tv, int lane, int q, int self, int cnt,
                           int K, float two_e, float& thr) {
  if (thr < 0.f || cnt < K) return 0;
  const GrpCut f = grp_tighten<S>(w.bs[q], w.bi[q], lane, cnt, K, 0, two_e);
  // every particle within the bound must have been taken, and every neighbour must be
  // provably at a non-zero distance: sqrt(s) (1 - 2^-20) > 2E
  const float zero2 = __fmul_ru(__fmul_ru(two_e, two_e), 1.01f);
  if (f.thr < 0.f || f.thr > thr || f.smin <= zero2 || f.cnt > 32 * S + 32) return 0;
  thr = f.thr;
  if (f.cnt == K) return 1;
  grp_drop<S>(w.bi[q], tv.pos, lane, self, f.cnt, K);
  return 2;
}

// The group's density sums (CalcDensity, KDCalcSmoothQuantities.cxx:260-286): okm marks the
// queries answered here, bi their neighbours. SAVE: the neighbour rows are kept too, the
// farthest last.
template <int S, bool SAVE>
__device__ void grp_density(const KnnArgs& a, const TreeView& tv, GrpSmem<S>& w, int lane, int gs,
                            unsigned okm, int K) {
  const unsigned FULL = 0xffffffffu;
  const int kr = a.kernres;
  const double* T = a.kernel;
  long long top = 0;
#pragma unroll 1
  for (unsigned left = okm; left; left &= left - 1) {
    const int q = __ffs(left) - 1;
    const P4 x = tv.pos[gs + q];
    double* row = reinterpret_cast<double*>(w.bs[q]);
    double d2[S];
    long long mx = 0;
#pragma unroll
    for (int s = 0; s < S; s++) {
      const int p = s * 32 + lane;
      d2[s] = kGrpNone;
      if (p < K) {
        const P4 c = tv.pos[w.bi[q][p]];
        const double dx = dsub(x.x, c.x), dy = dsub(x.y, c.y), dz = dsub(x.z, c.z);
        d2[s] = __fma_rn(dz, dz, __fma_rn(dy, dy, dmul(dx, dx)));
        mx = max(mx, dkey(d2[s]));
      }
    }
    mx = warp_max_key(mx);
    if (lane == q) top = mx;
    int at = K - 1;  // where the farthest is
#pragma unroll
    for (int s = S - 1; s >= 0; s--) {
      const bool is = dkey(d2[s]) == mx;
      if (SAVE) {
        const unsigned b = __ballot_sync(FULL, is);
        if (b) at = s * 32 + __ffs(b) - 1;
      }
      row[s * 32 + lane] = is ? kGrpFar : d2[s];
    }
    if (SAVE) {
#pragma unroll
      for (int s = 0; s < S; s++) {
        const int p = s * 32 + lane;
        if (p < K)
          a.nn[(size_t)(gs + q - tv.pstart) * K + (p == at ? K - 1 : (p == K - 1 ? at : p))] =
              w.bi[q][p];
      }
    }
  }
  // a lane per query: 1/h (h = sqrt(top) / 2), the table coordinate's scale, the weights
  double c1 = 0.0, wn = 0.0, wm = 0.0;
  if ((okm >> lane) & 1u) {
    const double ih = two_rsqrt(__longlong_as_double(top));
    c1 = dmul(ih, 0.5 * (double)(kr - 1));
    wn = 0.5 * dmul(dmul(ih, ih), ih);
    wm = dmul(wn, tv.pos[gs + lane].m);
  }
  __syncwarp();
  grp_sums<S>(w.bs, w.bi, tv.pos, a.rho + gs, a.rho, T, kr, lane, okm, K, c1, wn, wm);
}

// The group's velocity densities (CalcVelDensity, KDCalcSmoothQuantities.cxx:354-383): the
// nsmooth smallest |dv| of the neighbours, h = 0.5 max, sum Wsm(|dv|/h) h^-3, unit weights.
template <int S>
__device__ void grp_veldensity(const KnnArgs& a, const TreeView& tv, GrpSmem<S>& w, int lane,
                               int gs, unsigned okm, int K) {
  const unsigned FULL = 0xffffffffu;
  const int kr = a.kernres, ns = a.nsmooth;
  const double* T = a.kernel;
  long long top = 0;
#pragma unroll 1
  for (unsigned left = okm; left; left &= left - 1) {
    const int q = __ffs(left) - 1;
    const V4 x = tv.vel[gs + q];
    double* row = reinterpret_cast<double*>(w.bs[q]);
    long long vk[S];
#pragma unroll
    for (int s = 0; s < S; s++) {
      const int p = s * 32 + lane;
      vk[s] = kWqSent;
      if (p < K) {
        const V4 c = tv.vel[w.bi[q][p]];
        const double dx = dsub(x.x, c.x), dy = dsub(x.y, c.y), dz = dsub(x.z, c.z);
        vk[s] = dkey(__fma_rn(dz, dz, __fma_rn(dy, dy, dmul(dx, dx))));
      }
    }
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
    long long mx = 0;
#pragma unroll
    for (int s = 0; s < S; s++)
      if (sel[s]) mx = max(mx, vk[s]);
    mx = warp_max_key(mx);
    if (lane == q) top = mx;
#pragma unroll
    for (int s = 0; s < S; s++)
      row[s * 32 + lane] =
          !sel[s] ? kGrpNone : (vk[s] == mx ? kGrpFar : __longlong_as_double(vk[s]));
  }
  double c1 = 0.0, wn = 0.0;
  if ((okm >> lane) & 1u) {
    const double ih = two_rsqrt(__longlong_as_double(top));
    c1 = dmul(ih, 0.5 * (double)(kr - 1));
    wn = dmul(dmul(ih, ih), ih);
  }
  __syncwarp();
#pragma unroll 1
  for (unsigned left = okm; left; left &= left - 1) {
    const int q = __ffs(left) - 1;
    const double c = __shfl_sync(FULL, c1, q);
    double* row = reinterpret_cast<double*>(w.bs[q]);
#pragma unroll
    for (int s = 0; s < S; s++) row[s * 32 + lane] = grp_w(row[s * 32 + lane], c, kr, T);
  }
  __syncwarp();
  const double acc = grp_row_sums<S>(w.bs, lane);
  constexpr int lanes = 32 / GrpCfg<S>::G;
  const int q = lane / lanes;
  const double n = __shfl_sync(FULL, wn, q);
  if (lane % lanes == 0 && ((okm >> q) & 1u)) a.vden[gs + q] = dmul(acc, n);
  __syncwarp();
}

// One query's neighbour row, the farthest last. The FP32 squared distances name it unless
// another one is within their rounding of it; then FP64 distances do.
template <int S>
__device__ __forceinline__ void grp_save(const KnnArgs& a, const TreeView& tv, GrpSmem<S>& w,
                                         int lane, int q, int self, int how, int K, float two_e) {
  const unsigned FULL = 0xffffffffu;
  int idx[S];
  unsigned sb[S], mx = 0u;
#pragma unroll
  for (int s = 0; s < S; s++) {
    const int p = s * 32 + lane;
    idx[s] = p < K ? w.bi[q][p] : 0;
    sb[s] = p < K ? w.bs[q][p] : 0u;
    mx = max(mx, sb[s]);
  }
  mx = __reduce_max_sync(FULL, mx);
  int at = 0, c = 0;
#pragma unroll
  for (int s = 0; s < S; s++) {
    const unsigned b = __ballot_sync(
        FULL, s * 32 + lane < K &&
                  grp_thresh(__uint_as_float(sb[s]), two_e) >= __uint_as_float(mx));
    if (b) at = s * 32 + __ffs(b) - 1;
    c += __popc(b);
  }
  if (how == 2 || c != 1) {
    const P4 x = tv.pos[self];
    long long key[S], km = 0;
#pragma unroll
    for (int s = 0; s < S; s++) {
      key[s] = 0;
      if (s * 32 + lane < K) {
        const P4 y = tv.pos[idx[s]];
        key[s] = dkey(dist2_exact(x.x, x.y, x.z, y.x, y.y, y.z));
      }
      km = max(km, key[s]);
    }
    km = warp_max_key(km);
#pragma unroll
    for (int s = 0; s < S; s++) {
      const unsigned b = __ballot_sync(FULL, s * 32 + lane < K && key[s] == km);
      if (b) at = s * 32 + __ffs(b) - 1;
    }
  }
#pragma unroll
  for (int s = 0; s < S; s++) {
    const int p = s * 32 + lane;
    if (p < K)
      a.nn[(size_t)(self - a.q0) * K + (p == at ? K - 1 : (p == K - 1 ? at : p))] = idx[s];
  }
}

// The warp-per-query search for the queries the group kernel left: a persistent grid over
// the list fb[1 .. fb[0]] of tree indices.
template <int S, int EPI>
__global__ void __launch_bounds__(32 * kWqWpb, 4) k_knn_wq_list(KnnArgs a) {
  __shared__ WqSmem ws[kWqWpb];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int count = min(a.fb[0], a.nq);
  for (int i = blockIdx.x * kWqWpb + warp; i < count; i += gridDim.x * kWqWpb) {
    const int self = a.fb[1 + i];
    P4 p = a.tv.pos[self];
    double x0[3] = {p.x, p.y, p.z};
    wq_run<S, EPI>(a, a.tv, ws[warp], lane, self - a.q0, self, x0, a.kheap);
    __syncwarp();
  }
}

// Queries of `mask` left to the second launch.
__device__ __forceinline__ void grp_leave(int* fb, int lane, int gs, unsigned mask) {
  if (!mask) return;
  int base = 0;
  if (lane == 0) base = atomicAdd(&fb[0], __popc(mask));
  base = __shfl_sync(0xffffffffu, base, 0);
  if ((mask >> lane) & 1u) fb[1 + base + __popc(mask & ((1u << lane) - 1u))] = gs + lane;
}

constexpr int kGrpImage = 28;  // an index's bits from here on: the image pass it was found in

// FindNearest on a periodic tree: the direct pass's K nearest, then the image passes in the
// reference's order with its gates (KDSplitNode.cxx:1126-1147), each for the queries of the
// group whose gate it opens. A gate compares the exact K-th distance with a wall distance; the
// bounds of the selection decide unless they straddle it (that query takes the second launch).
// The images of the queries are searched with offsets from one of them as the centre.
template <int S>
__device__ void grp_periodic(const KnnArgs& a, GrpSmem<S>& w, int lane, int g, int depth, int K) {
  const unsigned FULL = 0xffffffffu;
  const TreeView& tv = a.tv;
  GrpLane L;
  int gs, gn;
  float two_e;
  grp_search<S>(w, tv, lane, g, depth, K, L, gs, gn, two_e);
  // cut every buffer to the K nearest; `okm`: the queries answered here
  unsigned okm = 0u;
  auto cut = [&](unsigned which, bool direct) {
#pragma unroll 1
    for (unsigned left = which; left; left &= left - 1) {
      const int q = __ffs(left) - 1;
      const float thr = __shfl_sync(FULL, L.thr, q);
      const int cnt = __shfl_sync(FULL, L.cnt, q);
      okm &= ~(1u << q);
      if (thr < 0.f || cnt < K) continue;
      const GrpCut f = grp_tighten<S>(w.bs[q], w.bi[q], lane, cnt, K, 0, two_e);
      const float zero2 = __fmul_ru(__fmul_ru(two_e, two_e), 1.01f);
      if (f.thr < 0.f || f.cnt > 32 * S + 32 || (direct && (f.thr > thr || f.smin <= zero2)))
        continue;
      okm |= 1u << q;
      if (lane == q) {
        L.cnt = f.cnt;
        L.thr = fminf(thr, f.thr);
      }
    }
  };
  cut((1u << gn) - 1u, true);
  const bool mine = (okm >> lane) & 1u;
  float slack = 2.f * two_e;  // a bound's root is at most this and 2^-16 above the K-th distance
  double x0[3] = {0, 0, 0};
  int near_sq = 0, near_lin = 0;
  if (mine) {
    const P4 p = tv.pos[gs + lane];
    x0[0] = p.x;
    x0[1] = p.y;
    x0[2] = p.z;
    const float4 qf = tv.posf[gs + lane];
    const float qeps = __fmul_ru(2.f, tv.eps);
    near_sq = near_walls(qf, tv.period, qeps, L.thr);
    near_lin = near_walls_lin(qf, tv.period, qeps, L.thr);
  }
#pragma unroll 1
  for (int pass = 1; pass < 8; pass++) {
    const int mk = kImageMask[pass];
    const bool lin = !(pass <= 3 || a.min_image);
    bool open = ((okm >> lane) & 1u) && (mk & ~(lin ? near_lin : near_sq)) == 0;
    if (!__any_sync(FULL, open)) continue;
    double xp[3];
    const float sv = __double2float_rn(reflect(x0, xp, tv.period, mk));
    // the K-th distance is between lo and hi
    const float hi = __fsqrt_ru(L.thr);
    const float lo = fmaxf(0.f, hi * (1.0f - 1.0f / 65536.0f) - slack);
    const float t1 = lin ? lo * lo : lo, t2 = lin ? L.thr : hi;
    const float m = fabsf(sv) * 1e-6f;
    const bool surely = t1 > sv + m, never = t2 < sv - m;
    okm &= ~__ballot_sync(FULL, open && !surely && !never);  // too close to call
    open = open && surely;
    const unsigned om = __ballot_sync(FULL, open);
    if (!om) continue;
    GrpGeom ge;
    double c[3];
#pragma unroll
    for (int d = 0; d < 3; d++) c[d] = __shfl_sync(FULL, xp[d], __ffs(om) - 1);
    ge.ch = make_float4(__double2float_rn(c[0]), __double2float_rn(c[1]), __double2float_rn(c[2]), 0.f);
    ge.cl = make_float4(__double2float_rn(dsub(c[0], (double)ge.ch.x)),
                        __double2float_rn(dsub(c[1], (double)ge.ch.y)),
                        __double2float_rn(dsub(c[2], (double)ge.ch.z)), 0.f);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    L.act = open;
    if (open) {
      p = make_float4(__double2float_rn(xp[0]), __double2float_rn(xp[1]), __double2float_rn(xp[2]), 0.f);
      L.x = __double2float_rn(dsub(xp[0], c[0]));
      L.y = __double2float_rn(dsub(xp[1], c[1]));
      L.z = __double2float_rn(dsub(xp[2], c[2]));
      w.qs[lane] = make_float4(L.x, L.y, L.z, L.thr);
    }
    const float far = __uint_as_float(__reduce_max_sync(
        FULL, open ? __float_as_uint(fmaxf(fabsf(L.x), fmaxf(fabsf(L.y), fabsf(L.z)))) : 0u));
    const float here = __fmul_ru(4.f, __fadd_ru(__fmul_ru(far, 1.f / 4194304.f),
                                                __fmul_ru(tv.eps, 1.f / 524288.f)));
    if (here > two_e) {
      // these offsets are rounded more than those the bounds were formed with: the bounds
      // widen by as much, and so does what lies between them and the K-th distances
      two_e = here;
      slack = __fadd_ru(slack, 2.f * two_e);
      L.thr = grp_thresh(L.thr, two_e);
      if (open) w.qs[lane].w = L.thr;
    }
    grp_box<S>(ge, open, p, __fmul_ru(2.f, tv.eps));
    const float wide = __uint_as_float(__reduce_max_sync(FULL, open ? __float_as_uint(L.thr) : 0u));
    ge.reach = grp_thresh(wide, two_e);
    __syncwarp();
    if (!grp_walk<S>(w, tv, ge, L, lane, gs, 0, 0, pass << kGrpImage, K, two_e)) {
      okm &= ~om;
      continue;
    }
    cut(om, false);
  }
  // the exact distances, from the image each neighbour was found in; rows as kEpiNN's
  const int off = 1 - (a.kheap - (a.drop_largest ? 1 : 0) - a.kout);
#pragma unroll 1
  for (unsigned left = okm; left; left &= left - 1) {
    const int q = __ffs(left) - 1, cnt = __shfl_sync(FULL, L.cnt, q);
    double x[3];
#pragma unroll
    for (int d = 0; d < 3; d++) x[d] = __shfl_sync(FULL, x0[d], q);
    long long key[S + 1];
    int idx[S + 1];
    auto exact = [&](int id) {
      const int mk = kImageMask[id >> kGrpImage];
      double xp[3] = {x[0], x[1], x[2]};
      if (mk) reflect(x, xp, tv.period, mk);
      const P4 y = tv.pos[id & ((1 << kGrpImage) - 1)];
      return dkey(dist2_exact(xp[0], xp[1], xp[2], y.x, y.y, y.z));
    };
    __syncwarp();
#pragma unroll
    for (int s = 0; s <= S; s++) {
      const int p = s * 32 + lane;
      key[s] = 0;
      idx[s] = -1;
      if (p < cnt) {
        idx[s] = w.bi[q][p];
        key[s] = exact(idx[s]);
      }
    }
    if (cnt > K) {
      grp_keep<S>(key, idx, w.bi[q], lane, cnt, K);
#pragma unroll
      for (int s = 0; s < S; s++)
        if (s * 32 + lane < K) {
          idx[s] = w.bi[q][s * 32 + lane];
          key[s] = exact(idx[s]);
        }
    }
    long long kk[S];
    int jj[S];
#pragma unroll
    for (int s = 0; s < S; s++) {
      const bool in = s * 32 + lane < K;
      kk[s] = in ? key[s] : kWqSent;
      jj[s] = in ? idx[s] & ((1 << kGrpImage) - 1) : -1;
    }
    grp_sort<S>(kk, jj, lane);
    const size_t row = (size_t)(gs + q - a.q0) * a.kout;
#pragma unroll
    for (int s = 0; s < S; s++) {
      const int i = s * 32 + lane + off;
      if (s * 32 + lane < K && i >= 0 && i < a.kout) {
        a.nn[row + i] = jj[s];
        a.d2[row + i] = __longlong_as_double(kk[s]);
      }
    }
    if (off > 0 && lane == 0) {
      a.nn[row] = gs + q;
      a.d2[row] = 0.0;
    }
  }
  grp_leave(a.fb, lane, gs, ((1u << gn) - 1u) & ~okm);
}

// A group without images: its searches, then what EPI makes of the neighbours.
template <int S, int EPI>
__device__ __forceinline__ void grp_serve(const KnnArgs& a, const TreeView& tv, GrpSmem<S>& w,
                                          int lane, int g, int depth, int K) {
  const unsigned FULL = 0xffffffffu;
  GrpLane L;
  int gs, gn;
  float two_e;
  grp_search<S>(w, tv, lane, g, depth, K, L, gs, gn, two_e);
  unsigned okm = 0u;  // queries answered here; the others take the second launch
#pragma unroll 1
  for (int q = 0; q < gn; q++) {
    float thr = __shfl_sync(FULL, L.thr, q);
    const int cnt = __shfl_sync(FULL, L.cnt, q), self = gs + q;
    const int how = grp_select<S>(w, tv, lane, q, self, cnt, K, two_e, thr);
    if (how == 0) continue;
    okm |= 1u << q;
    if (EPI == kEpiSave) grp_save<S>(a, tv, w, lane, q, self, how, K, two_e);
    if (EPI == kEpiNN) {
      const P4 x = tv.pos[self];
      long long key[S];
      int idx[S];
#pragma unroll
      for (int s = 0; s < S; s++) {
        key[s] = kWqSent;
        idx[s] = -1;
        if (s * 32 + lane < K) {
          idx[s] = w.bi[q][s * 32 + lane];
          const P4 c = tv.pos[idx[s]];
          key[s] = dkey(dist2_exact(x.x, x.y, x.z, c.x, c.y, c.z));
        }
      }
      grp_sort<S>(key, idx, lane);
      // the row leaves out the nearest (FindNearest) or the largest (FindNearestPos) where one
      // more was asked
      const int off = -(a.kheap - (a.drop_largest ? 1 : 0) - a.kout);
      const size_t row = (size_t)(self - a.q0) * a.kout;
#pragma unroll
      for (int s = 0; s < S; s++) {
        const int i = s * 32 + lane + off;
        if (s * 32 + lane < K && i >= 0 && i < a.kout) {
          a.nn[row + i] = idx[s];
          a.d2[row + i] = __longlong_as_double(key[s]);
        }
      }
    }
  }
  __syncwarp();
  if (EPI == kEpiDensity || EPI == kEpiDensVel || EPI == kEpiDensSave)
    grp_density<S, EPI == kEpiDensSave>(a, tv, w, lane, gs, okm, K);
  if (EPI == kEpiDensVel || EPI == kEpiVel) grp_veldensity<S>(a, tv, w, lane, gs, okm, K);
  grp_leave(a.fb, lane, gs, ((1u << gn) - 1u) & ~okm);
}

// K: neighbours other than the query itself; a periodic search's k + 1 list is the query
// itself at zero distance, then the K = k nearest others (images included).
template <int S>
__global__ void __launch_bounds__(32 * kGrpWpb, 6) k_knn_group_periodic(KnnArgs a, int depth, int K) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GrpSmem<S>& w = reinterpret_cast<GrpSmem<S>*>(smem_raw)[threadIdx.x >> 5];
  const int g = blockIdx.x * kGrpWpb + (threadIdx.x >> 5);
  if (g < (1 << depth)) grp_periodic<S>(a, w, lane_id(), g, depth, K);
}

template <int S, int EPI>
__global__ void __launch_bounds__(32 * kGrpWpb, 7) k_knn_group(KnnArgs a, int depth, int K) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GrpSmem<S>& w = reinterpret_cast<GrpSmem<S>*>(smem_raw)[threadIdx.x >> 5];
  const int g = blockIdx.x * kGrpWpb + (threadIdx.x >> 5);
  if (g >= (1 << (depth - a.slices))) return;
  grp_serve<S, EPI>(a, a.tv, w, lane_id(), g + (a.slice << (depth - a.slices)), depth, K);
}

// ---- batched density: every particle of every tree of a forest, k = min(k, n_tree - 1)

// Last entry of the ascending v[0 .. n) that is <= x.
__device__ __forceinline__ int last_at_most(const int* v, int n, int x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (v[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

template <int S>
__global__ void __launch_bounds__(32 * kGrpWpb, 7) k_knn_group_batch(KnnArgs a, BatchArgs b) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GrpSmem<S>& w = reinterpret_cast<GrpSmem<S>*>(smem_raw)[threadIdx.x >> 5];
  const int lane = lane_id();
  const int i = blockIdx.x * kGrpWpb + (threadIdx.x >> 5);
  if (i >= b.ngroups) return;
  const int t = last_at_most(b.goff, b.ntrees, i);
  const TreeInfo ti = b.trees[t];
  TreeView tv = a.tv;
  tv.n = ti.n;
  tv.pstart = ti.pstart;
  tv.nbase = ti.nbase;
  const int K = min(a.kheap, ti.n - 1), q = (ti.n - 1) / b.gmax;
  if (K < 1) return;
  // squares could leave the FP32 range: everything takes the list (as group_search_serves)
  if (tv.eps >= 1e11f || tv.eps <= 1e-19f) {
    if (i == b.goff[t])
      for (int p = lane; p < ti.n; p += 32) a.fb[1 + atomicAdd(&a.fb[0], 1)] = ti.pstart + p;
    return;
  }
  grp_serve<S, kEpiDensity>(a, tv, w, lane, i - b.goff[t], 32 - __clz(q), K);
}

// The batch's queries that the group kernel left (as k_knn_wq_list), each in its own tree.
template <int S>
__global__ void __launch_bounds__(32 * kWqWpb, 4) k_knn_wq_list_batch(KnnArgs a, BatchArgs b) {
  __shared__ WqSmem ws[kWqWpb];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int count = min(a.fb[0], a.nq);
  for (int i = blockIdx.x * kWqWpb + warp; i < count; i += gridDim.x * kWqWpb) {
    const int self = a.fb[1 + i];
    const TreeInfo ti = b.trees[last_at_most(b.pstart, b.ntrees, self)];
    TreeView tv = a.tv;
    tv.n = ti.n;
    tv.pstart = ti.pstart;
    tv.nbase = ti.nbase;
    P4 p = tv.pos[self];
    double x0[3] = {p.x, p.y, p.z};
    wq_run<S, kEpiDensity>(a, tv, ws[warp], lane, self, self, x0, min(a.kheap, ti.n - 1));
    __syncwarp();
  }
}

template <int S>
int launch_group_batch(const KnnArgs& a, const BatchArgs& b, cudaStream_t st) {
  const size_t sm = sizeof(GrpSmem<S>) * kGrpWpb;
  NBK_TRY(ensure_dyn_smem((const void*)k_knn_group_batch<S>, (int)sm));
  NBK_CUDA_TRY(cudaMemsetAsync(a.fb, 0, sizeof(int), st));
  if (b.ngroups == 0) return NBK_OK;
  Phase ph("knn_density_batch", st);
  k_knn_group_batch<S><<<(b.ngroups + kGrpWpb - 1) / kGrpWpb, 32 * kGrpWpb, sm, st>>>(a, b);
  note_launch();
  const unsigned lb = (unsigned)std::min<int64_t>(4 * b.nsm, ((int64_t)a.nq + kWqWpb - 1) / kWqWpb);
  k_knn_wq_list_batch<S><<<lb, 32 * kWqWpb, 0, st>>>(a, b); note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  return NBK_OK;
}

template <int S, int EPI>
int launch_group(const KnnArgs& a, int K, cudaStream_t st) {
  // groups of at most G particles, and enough of them to keep every SM's warps busy
  int nsm = 0, dev = 0;
  NBK_CUDA_TRY(cudaGetDevice(&dev));
  NBK_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  int depth = 0;
  const int64_t n = a.tv.n;
  while (((n - 1) >> depth) + 1 > GrpCfg<S>::G) depth++;
  while ((1 << depth) < 16 * nsm && ((n - 1) >> (depth + 1)) + 1 >= 2) depth++;
  const size_t sm = sizeof(GrpSmem<S>) * kGrpWpb;
  NBK_TRY(ensure_dyn_smem((const void*)k_knn_group<S, EPI>, (int)sm));
  static const char* kNames[] = {"knn_nn", "knn_density", "knn_density_veldensity", "knn_veldensity",
                                 "knn_density_particle", "knn_veldensity_particle", "knn_density_save",
                                 "knn_save"};
  NBK_CUDA_TRY(cudaMemsetAsync(a.fb, 0, sizeof(int), st));
  Phase ph(kNames[EPI], st);
  const unsigned blocks = ((1u << (depth - a.slices)) + kGrpWpb - 1) / kGrpWpb;
  if (EPI == kEpiNN && a.periodic) {
    NBK_TRY(ensure_dyn_smem((const void*)k_knn_group_periodic<S>, (int)sm));
    k_knn_group_periodic<S><<<blocks, 32 * kGrpWpb, sm, st>>>(a, depth, K); note_launch();
  } else {
    k_knn_group<S, EPI><<<blocks, 32 * kGrpWpb, sm, st>>>(a, depth, K); note_launch();
  }
  const unsigned lb = (unsigned)std::min<int64_t>(4 * nsm, ((int64_t)a.nq + kWqWpb - 1) / kWqWpb);
  if (a.kheap <= 32) k_knn_wq_list<1, EPI><<<lb, 32 * kWqWpb, 0, st>>>(a);
  else if (a.kheap <= 64) k_knn_wq_list<2, EPI><<<lb, 32 * kWqWpb, 0, st>>>(a);
  else k_knn_wq_list<4, EPI><<<lb, 32 * kWqWpb, 0, st>>>(a);
  note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  return NBK_OK;
}

template <int EPI>
int launch_group_e(const KnnArgs& a, cudaStream_t st) {
  const int K = a.periodic ? a.kheap - 1 : a.kheap;  // neighbours other than the query
  if (K <= 32) return launch_group<1, EPI>(a, K, st);
  if (K <= 64) return launch_group<2, EPI>(a, K, st);
  return launch_group<4, EPI>(a, K, st);
}

}  // namespace

// Particles per group of a batch: the largest of 8, 4 and 2 that the buffers for k take and
// that leaves enough groups to keep every SM's warps busy (index into the prefix arrays):
// a larger group shares one walk of the tree, a smaller one shortens what the last warp does
// (64 trees of 20 to 2000 particles, k = 32: 0.099 ms in groups of 8, 0.091 in smaller ones).
int batch_group_size(int k, const int64_t ngroups[3], int nsm) {
  int i = k <= 32 ? 0 : k <= 64 ? 1 : 2;
  while (i < 2 && ngroups[i] < 16 * nsm) i++;
  return i;
}

int launch_knn_group_batch(const KnnArgs& a, const BatchArgs& b, cudaStream_t st) {
  if (a.kheap <= 32) return launch_group_batch<1>(a, b, st);
  if (a.kheap <= 64) return launch_group_batch<2>(a, b, st);
  return launch_group_batch<4>(a, b, st);
}

// From how many particles on the groups are faster than a warp per query, where the particles
// lie evenly and where they are clustered (k_mixed, build.cu). A group's warp serves its queries
// one after another, and a group that lies partly in a much denser place takes many times as
// long as the others: fewer groups than the SMs have room for hide neither. The search's own work
// decides where: the sums cost a group less than its queries alone, sorted rows and image passes
// do not, and a warp per query holds more than 64 neighbours in four slots.
// Measured (time of a warp per query over the groups' time, k = 8, 32, 64; uniform, normal,
// Plummer sphere, 500 spheres, 8 spheres in a background):
//   density   16,384: 1.29 1.14 1.60, 1.22 1.07 1.16, 1.03 0.76 0.85, 0.94 0.91 0.88, 0.84 0.71 0.77
//             49,152: 1.68 1.80 1.58, 1.50 1.47 1.39, 1.27 1.12 1.13, 1.06 1.08 1.13, 0.91 0.87 0.95
//   rows      24,576: 1.33 1.25 1.30, 1.06 1.06 1.08, 0.88 0.81 0.81, 0.74 0.65 0.74, 0.68 0.64 0.72
//             98,304: 1.50 1.91 1.50, 1.43 1.53 1.25, 1.28 1.27 1.19, 1.02 1.07 1.07, 0.98 0.91 0.91
//   images    32,768: 1.13 1.12, 0.92 1.10, 0.71 0.78, 0.82 0.83, 0.65 0.81 (k = 8 and 32)
//             98,304: 1.41 1.79, 1.34 1.64, 1.25 1.31, 1.09 1.19, 1.03 1.00
//    k = 48   65,536: 1.18, 1.15, 0.95, 0.87, 0.71; 131,072: 1.25, 1.20, 1.10, 0.92, 0.93
//   k = 100    8,192: density 5.17 uniform, 2.25 in 500 spheres, 1.25 in 8; images 2.48, 1.54, 1.03
namespace {
struct GroupLines {
  int even, mixed;
};
GroupLines group_lines(const KnnArgs& a, int epi) {
  if (a.kheap > 64) return {kGroupSmallest, kGroupSmallest};
  if (epi != kEpiNN) return {kGroupMixedMin, 49152};
  if (!a.periodic) return {24576, 98304};
  return a.kheap <= 33 ? GroupLines{32768, 98304} : GroupLines{65536, kGroupMixedMax};
}
}  // namespace

// Every particle of a tree (or a slice of it), none of them given zero-distance or image
// answers that FP32 offsets cannot tell apart, k within the buffers, squares inside FP32 (below
// 1e-12 the neighbours' are not, and nearly every query would take the list: density of 2^20
// particles in a box of 1e-14 7.4 ms by groups, 5.8 a warp each).
bool group_search_serves(const KnnArgs& a, int epi) {
  const int K = a.periodic ? a.kheap - 1 : a.kheap;
  return a.qmode == 0 && (a.nq == a.tv.n || a.slices > 0) && a.kheap <= 128 && K >= 1 &&
         a.tv.n >= (a.mixed ? group_lines(a, epi).mixed : group_lines(a, epi).even) &&
         a.tv.eps < 1e11f && a.tv.eps > 1e-19f &&
         (a.periodic ? a.tv.n <= (1 << kGrpImage) : a.exclude_self != 0);
}

int launch_knn_group(const KnnArgs& a, int epi, cudaStream_t st) {
  switch (epi) {
    case kEpiNN: return launch_group_e<kEpiNN>(a, st);
    case kEpiDensity: return launch_group_e<kEpiDensity>(a, st);
    case kEpiDensVel: return launch_group_e<kEpiDensVel>(a, st);
    case kEpiVel: return launch_group_e<kEpiVel>(a, st);
    case kEpiDensSave: return launch_group_e<kEpiDensSave>(a, st);
    case kEpiSave: return launch_group_e<kEpiSave>(a, st);
  }
  set_error("unknown kNN epilogue");
  return NBK_ERR_INVALID;
}

}  // namespace nbk
