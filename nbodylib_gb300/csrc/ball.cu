// Fixed-radius searches (replaces KDTree::SearchBallPosTagged / SearchBallPos and their
// node recursions, src/KDTree/KDFindNearest.cxx:567-706, KDSplitNode.cxx:455-686,
// 1341-1456, KDLeafNode.cxx:247-410).
//
// One warp serves up to 32 queries and walks the tree once for them. Results are returned as
// CSR: a counting pass, an exclusive scan, a filling pass; a row lists its particles in tree
// order, image by image. Pair decisions are the reference's FP64 test d2 < fdist2 (strict);
// the whole-node shortcut of the reference marks exactly the particles this test accepts
// (every member of a node whose farthest corner is inside the radius passes it, because
// rounding is monotone), so it changes only whether the target itself is reported, which
// nbk_ball_mark reproduces from the exact node boxes.
//
// What bounds it: instruction issue. A lane per query tested every particle of an opened leaf
// for the whole warp, with two directed-rounding bounds, one node at a time (2.45 ms for 2^20
// balls of 32 in a uniform box, half the lanes idle). Now up to 32 nodes are taken at once
// (in tree order: the leaves ahead of the first inner node are tested, what follows is pushed
// back), leaf particles are tested a lane each, two leaves at a time, one query after another
// of those that want the leaf, and one round-to-nearest distance decides outside a band of
// its own rounding error around the radius (FP64 for all where squares leave FP32's range,
// fp32_band): 1.50 ms (both passes; 32 warps per SM at 64 registers and some 70 bytes of spills;
// with 40, which spill more, 1.53 ms).
#include "nbk_build.h"

namespace nbk {

namespace {

constexpr int kStack = 512;  // node stack of one warp
constexpr int kBatch = kStack - 128;
constexpr int kWpb = 4;
// Volume in cubed radii of the box around a warp's balls above which nodes are tested query by
// query: 32 balls apart from one another fill 134. (2^17 targets in random order of 2^20
// particles, 32 per ball: 98 ms never tested, 1.28 with this line; 20,001 targets with 64 per
// ball: 1.32 never, 0.66 with the line at 512, 0.24 at 128; 2^20 in tree order 1.55 either way,
// 1.86 always tested.)
constexpr float kBallVolume = 128.f;

struct BallArgs {
  TreeView tv;
  int qmode;  // 0: targets (tree indices), 1: coordinates
  const int* qidx;
  const double* qx;
  int nq;
  int qpw;    // queries per warp
  double r2;
  int exclude_self;
  int* counts;
  const int64_t* offsets;
  int* out;
  double* outd2;
  int* err;
};

struct BallSmem {
  float4 q[32];  // the warp's query points of this pass (FP32)
  int stk[kStack];
};

template <bool FILL>
__global__ void __launch_bounds__(32 * kWpb, 8) k_ball(BallArgs a) {
  __shared__ BallSmem sm[kWpb];
  const unsigned FULL = 0xffffffffu;
  int lane;  // read once
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  const int warp = threadIdx.x >> 5;
  BallSmem& w = sm[warp];
  const TreeView& tv = a.tv;
  const int q0 = (blockIdx.x * kWpb + warp) * a.qpw, q = q0 + lane;
  if (q0 >= a.nq) return;
  const bool valid = lane < a.qpw && q < a.nq;
  int self = -1;
  double x0[3] = {0, 0, 0};
  if (valid) {
    if (a.qmode == 0) {
      self = a.qidx[q];
      P4 p = tv.pos[self];
      x0[0] = p.x;
      x0[1] = p.y;
      x0[2] = p.z;
    } else {
      x0[0] = a.qx[3 * (size_t)q];
      x0[1] = a.qx[3 * (size_t)q + 1];
      x0[2] = a.qx[3 * (size_t)q + 2];
    }
  }
  const int64_t base = (FILL && valid) ? a.offsets[q] : 0;
  const int room = (FILL && valid) ? (int)(a.offsets[q + 1] - base) : 0;
  int cnt = 0;
  const float thr = thresh_hi(a.r2), r2_lo = thresh_lo(a.r2);
  const long long r2k = a.r2 > 0.0 ? dkey(a.r2) : 0;  // nothing is inside r2 <= 0 or NaN
  // the query's own rounding bound, images included (it may lie outside the tree's box)
  const float eps = valid ? query_eps(tv, x0[0], x0[1], x0[2]) : tv.eps;
  // |sqrt(s) - d| <= e + 2^-21 d for the round-to-nearest s of a pair at distance d (the
  // coordinate differences are off by eps + tv.eps each; the warp's largest)
  float e = eps;
  for (int o = 16; o > 0; o >>= 1) e = fmaxf(e, __shfl_xor_sync(FULL, e, o));
  const Band band = fp32_band(__fsqrt_ru(thr), __fsqrt_rd(r2_lo),
                              __fmul_ru(__fadd_ru(e, tv.eps), 1.7321f), 1.0f / 524288.0f);
  const float far2 = band.far2, near2 = band.near2;
  const int npass = tv.periodic ? 8 : 1;
  int near = 0;
  if (tv.periodic && valid)
    near = near_walls(make_float4(__double2float_rn(x0[0]), __double2float_rn(x0[1]),
                                  __double2float_rn(x0[2]), 0.f),
                      tv.period, eps, thr);
  for (int pass = 0; pass < npass; pass++) {
    double xq[3] = {x0[0], x0[1], x0[2]};
    bool active = valid;
    if (pass > 0) {
      const bool may = valid && (kImageMask[pass] & ~near) == 0;
      if (!__any_sync(FULL, may)) continue;
      const double sval = reflect(x0, xq, tv.period, kImageMask[pass]);
      active = may && (a.r2 > dmul(sval, sval));  // KDSplitNode.cxx:1356-1373
    }
    if (!__any_sync(FULL, active)) continue;
    const float qx = __double2float_rn(xq[0]), qy = __double2float_rn(xq[1]),
                qz = __double2float_rn(xq[2]);
    // box around the active lanes' query points, widened by their rounding; where it is much
    // larger than their balls together (points in no order, or on both sides of a high split)
    // nodes are taken only if a ball reaches them
    float qlo[3], qhi[3], vol = 1.f;
    {
      const float v[3] = {qx, qy, qz};
#pragma unroll
      for (int d = 0; d < 3; d++) {
        float lo = active ? __fsub_rd(v[d], eps) : FLT_MAX;
        float hi = active ? __fadd_ru(v[d], eps) : -FLT_MAX;
        for (int o = 16; o > 0; o >>= 1) {
          lo = fminf(lo, __shfl_xor_sync(FULL, lo, o));
          hi = fmaxf(hi, __shfl_xor_sync(FULL, hi, o));
        }
        qlo[d] = lo;
        qhi[d] = hi;
        vol *= (hi - lo) * rsqrtf(thr) + 2.f;
      }
    }
    const bool strict = !(vol <= kBallVolume);  // infinite or NaN: an empty ball
    __syncwarp();
    w.q[lane] = make_float4(qx, qy, qz, 0.f);
    if (lane == 0) w.stk[0] = 0;
    int sp = 1;
    __syncwarp();
#pragma unroll 1
    while (sp > 0) {
      // the next nodes in tree order, the first on lane 0; above kBatch entries one at a time
      // (a depth-first descent from there adds at most the tree depth). A node that has been
      // tested is stored as its complement.
      const int m = sp <= kBatch ? min(32, sp) : 1;
      int h = -1;
      NodeRec r{};
      bool keep = false;
      if (lane < m) {
        h = w.stk[sp - 1 - lane];
        keep = h < 0;
        h = h < 0 ? ~h : h;
        r = tv.node[tv.nbase + h];
        if (!keep) {
          const float gx = fmaxf(0.f, fmaxf(__fsub_rd(r.lo[0], qhi[0]), __fsub_rd(qlo[0], r.hi[0])));
          const float gy = fmaxf(0.f, fmaxf(__fsub_rd(r.lo[1], qhi[1]), __fsub_rd(qlo[1], r.hi[1])));
          const float gz = fmaxf(0.f, fmaxf(__fsub_rd(r.lo[2], qhi[2]), __fsub_rd(qlo[2], r.hi[2])));
          keep = __fadd_rd(__fadd_rd(__fmul_rd(gx, gx), __fmul_rd(gy, gy)), __fmul_rd(gz, gz)) < thr;
        }
      }
      __syncwarp();
      sp -= m;
      const bool leaf = r.count <= tv.b;
      if (strict) {
        // a lane per node, as far as a hit of any query can be (see far2; outside
        // FP32's range every node)
        bool reach = false;
#pragma unroll 1
        for (unsigned qm = __ballot_sync(FULL, active); qm; qm &= qm - 1) {
          const float4 qf = w.q[__ffs(qm) - 1];
          const float gx = fmaxf(0.f, fmaxf(r.lo[0] - qf.x, qf.x - r.hi[0]));
          const float gy = fmaxf(0.f, fmaxf(r.lo[1] - qf.y, qf.y - r.hi[1]));
          const float gz = fmaxf(0.f, fmaxf(r.lo[2] - qf.z, qf.z - r.hi[2]));
          reach = reach || !(gx * gx + gy * gy + gz * gz >= far2);
        }
        keep = keep && reach;
      }
      const unsigned km = __ballot_sync(FULL, keep), im = __ballot_sync(FULL, keep && !leaf);
      const unsigned ahead = im ? (im & (0u - im)) - 1u : 0xffffffffu;  // lanes before it
      // what follows the first inner node goes back, its children in its place
      const unsigned back = km & ~ahead, two = back & im;
      const int up = 31 - lane;  // lanes after this one
      const int slot = sp + (up ? __popc(back >> (lane + 1)) + __popc(two >> (lane + 1)) : 0);
      const int total = __popc(back) + __popc(two);
      if (sp + total > kStack) {
        if (lane == 0) atomicExch(a.err, kErrCapacity);
        return;
      }
      if ((back >> lane) & 1u) {
        if (leaf) {
          w.stk[slot] = ~h;
        } else {
          w.stk[slot] = 2 * h + 2;
          w.stk[slot + 1] = 2 * h + 1;
        }
      }
      sp += total;
      // the leaves ahead, two at a time
      unsigned lm = km & ahead;
#pragma unroll 1
      while (lm) {
        int st = 0, ct = 0;
        unsigned mk = 0, any = 0;
#pragma unroll
        for (int half = 0; half < 2; half++) {
          if (!lm) break;
          const int j = __ffs(lm) - 1;
          NodeRec rj;
#pragma unroll
          for (int d = 0; d < 3; d++) {
            rj.lo[d] = __shfl_sync(FULL, r.lo[d], j);
            rj.hi[d] = __shfl_sync(FULL, r.hi[d], j);
          }
          const int cj = __shfl_sync(FULL, r.count, j), sj = __shfl_sync(FULL, r.start, j);
          if (half == 1 && (cj > 16 || __any_sync(FULL, ct > 16))) break;  // a row stays in order
          lm &= lm - 1;
          const unsigned nm =
              __ballot_sync(FULL, active && box_d2_lo(qx, qy, qz, eps, rj) < thr);
          if ((lane >> 4) == half) {
            st = sj;
            ct = cj;
            mk = nm;
          }
          any |= nm;
        }
        if (!any) continue;
        const bool big = __any_sync(FULL, ct > 16);  // one leaf alone, 32 particles a step
        if (big) {
          st = __shfl_sync(FULL, st, 0);
          ct = __shfl_sync(FULL, ct, 0);
          mk = any;
        }
        const int step = big ? 32 : 16, off = big ? lane : (lane & 15);
#pragma unroll 1
        for (; __any_sync(FULL, ct > 0); st += step, ct -= step) {
          const int ti = st + off;
          const bool ok = off < ct;
          float4 cf = make_float4(0.f, 0.f, 0.f, 0.f);
          if (ok) cf = tv.posf[ti];
#pragma unroll 1
          for (unsigned qm = any; qm; qm &= qm - 1) {
            const int i = __ffs(qm) - 1;
            const float4 qf = w.q[i];
            const float dx = cf.x - qf.x, dy = cf.y - qf.y, dz = cf.z - qf.z;
            const float s = dx * dx + dy * dy + dz * dz;
            bool in = ok && ((mk >> i) & 1u) && !(s >= far2);
            const int si = __shfl_sync(FULL, self, i);
            if (a.exclude_self && pass == 0) in = in && ti != si;
            const bool open = in && (!(s < near2) || (FILL && a.outd2));
            double d2 = 0.0;
            if (__any_sync(FULL, open)) {
              double xi[3];
#pragma unroll
              for (int d = 0; d < 3; d++) xi[d] = __shfl_sync(FULL, xq[d], i);
              if (open) {
                const P4 c = tv.pos[ti];
                d2 = dist2_exact(xi[0], xi[1], xi[2], c.x, c.y, c.z);
                in = dkey(d2) < r2k;  // d2 < r2
              }
            }
            const unsigned hit = __ballot_sync(FULL, in);
            if (FILL && hit) {
              const int64_t bi = __shfl_sync(FULL, base, i);
              const int c = __shfl_sync(FULL, cnt, i) + __popc(hit & ((1u << lane) - 1u));
              const int lim = __shfl_sync(FULL, room, i);
              if (in) {
                if (c < lim) {
                  a.out[bi + c] = ti;
                  if (a.outd2) a.outd2[bi + c] = d2;
                } else {
                  atomicExch(a.err, kErrCapacity);  // fill disagrees with count
                }
              }
            }
            if (lane == i) cnt += __popc(hit);
          }
        }
      }
      __syncwarp();
    }
  }
  if (!FILL && valid) a.counts[q] = cnt;
}

// Queries per warp: 32 where that leaves enough warps for every SM (a lane each; the other
// lanes still take nodes and particles). 16,385 balls of 32: 0.28 ms with 32 a warp, 0.22 with
// the 4 of this rule; 55,839 of 39: 0.41 and 0.36 with 16.
int ball_qpw(int64_t nq, int* qpw) {
  int dev = 0, nsm = 0;
  NBK_CUDA_TRY(cudaGetDevice(&dev));
  NBK_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  *qpw = 32;
  while (*qpw > 1 && nq / *qpw < 16 * nsm) *qpw /= 2;
  return NBK_OK;
}

__global__ void k_scan64_blocks(const int* in, int64_t* out, int64_t* bsum, int n) {
  __shared__ int64_t s[1024];
  int i = blockIdx.x * 1024 + threadIdx.x;
  int64_t v = i < n ? in[i] : 0;
  s[threadIdx.x] = v;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    int64_t t = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
    __syncthreads();
    s[threadIdx.x] += t;
    __syncthreads();
  }
  if (i < n) out[i] = s[threadIdx.x] - v;
  if (threadIdx.x == 1023) bsum[blockIdx.x] = s[1023];
}
__global__ void k_scan64_sums(int64_t* bsum, int nb, int64_t* total) {
  __shared__ int64_t s[1024];
  __shared__ int64_t run;
  if (threadIdx.x == 0) run = 0;
  __syncthreads();
  for (int c0 = 0; c0 < nb; c0 += 1024) {
    int i = c0 + threadIdx.x;
    int64_t v = i < nb ? bsum[i] : 0;
    s[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      int64_t t = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
      __syncthreads();
      s[threadIdx.x] += t;
      __syncthreads();
    }
    if (i < nb) bsum[i] = run + s[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) run += s[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = run;
}
__global__ void k_scan64_add(int64_t* out, const int64_t* bsum, int n, const int64_t* total) {
  int i = blockIdx.x * 1024 + threadIdx.x;
  if (i < n) out[i] += bsum[blockIdx.x];
  if (i == 0) out[n] = *total;
}

// Whether SearchBallPos(tt) reports the target: a node on the root-to-leaf path is
// flagged by FlagNodeForSearchBallPos (split nodes, KDNode.h:325-332 with
// __checkboundaries :280-291) or the leaf's whole-bucket test holds (KDLeafNode.cxx:
// 250-255), all in FP64 on the exact node boxes.
__global__ void k_mark(TreeView tv, int target, double r2, int imark, const int* found,
                       const double* found_d2, const int64_t* nfound, const int* perm,
                       int* mark, double* dist2, int check_self) {
  int64_t nf = *nfound;
  for (int64_t i = threadIdx.x + blockIdx.x * (int64_t)blockDim.x; i < nf;
       i += (int64_t)blockDim.x * gridDim.x) {
    int id = perm[found[i]];
    mark[id] = imark;
    dist2[id] = found_d2[i];
  }
  if (!check_self || blockIdx.x != 0 || threadIdx.x != 0) return;
  P4 p = tv.pos[target];
  double x[3] = {p.x, p.y, p.z};
  int h = 0;
  bool inc = false;
  for (int depth = 0; depth < 64; depth++) {
    const NodeX& nx = tv.nodex[tv.nbase + h];
    const NodeRec& r = tv.node[tv.nbase + h];
    bool leaf = r.count <= tv.b;
    double me = 0.0;
    for (int d = 0; d < 3; d++) me = fmax(me, dsub(nx.hi[d], nx.lo[d]));
    double maxr2 = 0.0;
    for (int d = 0; d < 3; d++) {
      double da = dsub(x[d], nx.lo[d]), db = dsub(nx.hi[d], x[d]);
      double a2 = dmul(da, da), b2 = dmul(db, db);
      maxr2 = dadd(maxr2, a2 > b2 ? a2 : b2);
    }
    if (leaf) {
      inc = maxr2 < r2;
      break;
    }
    if (!(dmul(me, me) > r2) && maxr2 < r2) {
      inc = true;
      break;
    }
    const NodeRec& l = tv.node[tv.nbase + 2 * h + 1];
    h = (target < l.start + l.count) ? 2 * h + 1 : 2 * h + 2;
  }
  if (inc) {
    int id = perm[target];
    mark[id] = imark;
    dist2[id] = 0.0;
  }
}

}  // namespace

int run_ball(const TreeView& tv, int qmode, const int* qidx, const double* qx, int nq,
             double fdist2, int exclude_self, int64_t* d_offsets, int* d_out,
             int64_t out_capacity, int64_t* h_total, DevAlloc& alloc, cudaStream_t st) {
  if (nq == 0) {
    *h_total = 0;
    NBK_CUDA_TRY(cudaMemsetAsync(d_offsets, 0, sizeof(int64_t), st));
    return NBK_OK;
  }
  int* counts;
  int64_t *bsum, *d_total;
  int* err;
  int nb = (nq + 1023) / 1024;
  NBK_TRY(alloc.get((void**)&counts, sizeof(int) * nq));
  NBK_TRY(alloc.get((void**)&bsum, sizeof(int64_t) * (nb + 1)));
  NBK_TRY(alloc.get((void**)&d_total, sizeof(int64_t)));
  NBK_TRY(alloc.get((void**)&err, sizeof(int)));
  NBK_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
  BallArgs a{};
  a.tv = tv;
  a.qmode = qmode;
  a.qidx = qidx;
  a.qx = qx;
  a.nq = nq;
  a.r2 = fdist2;
  a.exclude_self = exclude_self;
  a.counts = counts;
  a.err = err;
  NBK_TRY(ball_qpw(nq, &a.qpw));
  const int64_t warps = ((int64_t)nq + a.qpw - 1) / a.qpw;
  const unsigned blocks = (unsigned)((warps + kWpb - 1) / kWpb);
  Phase ph("ball", st);
  k_ball<false><<<blocks, 32 * kWpb, 0, st>>>(a); note_launch();
  k_scan64_blocks<<<nb, 1024, 0, st>>>(counts, d_offsets, bsum, nq); note_launch();
  k_scan64_sums<<<1, 1024, 0, st>>>(bsum, nb, d_total); note_launch();
  k_scan64_add<<<nb, 1024, 0, st>>>(d_offsets, bsum, nq, d_total); note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  int64_t total = 0;
  int herr = 0;
  NBK_CUDA_TRY(cudaMemcpyAsync(&total, d_total, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  NBK_CUDA_TRY(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st));
  NBK_CUDA_TRY(cudaStreamSynchronize(st));
  *h_total = total;
  if (herr) {
    set_error("ball search: device traversal stack exceeded");
    return NBK_ERR_DEVICE;
  }
  if (total > out_capacity || d_out == nullptr) {
    set_error("ball search: output capacity " + std::to_string(out_capacity) + " < " +
              std::to_string(total) + " results");
    return NBK_ERR_INVALID;
  }
  a.offsets = d_offsets;
  a.out = d_out;
  a.outd2 = nullptr;
  k_ball<true><<<blocks, 32 * kWpb, 0, st>>>(a); note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  return NBK_OK;
}

int run_ball_mark(const TreeView& tv, int target, double fdist2, int imark, int* d_mark,
                  double* d_dist2, const int* d_perm, int target_search, cudaStream_t st) {
  DevAlloc alloc;
  int* d_t;
  int64_t* d_off;
  int* err;
  NBK_TRY(alloc.get((void**)&d_t, sizeof(int)));
  NBK_TRY(alloc.get((void**)&d_off, sizeof(int64_t) * 2));
  NBK_TRY(alloc.get((void**)&err, sizeof(int)));
  NBK_CUDA_TRY(cudaMemcpyAsync(d_t, &target, sizeof(int), cudaMemcpyHostToDevice, st));
  NBK_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
  // count
  BallArgs a{};
  a.tv = tv;
  a.qmode = 0;
  a.qidx = d_t;
  a.nq = 1;
  a.qpw = 1;
  a.r2 = fdist2;
  a.exclude_self = target_search;
  int* counts;
  NBK_TRY(alloc.get((void**)&counts, sizeof(int)));
  a.counts = counts;
  a.err = err;
  k_ball<false><<<1, 32 * kWpb, 0, st>>>(a); note_launch();
  int hc = 0;
  NBK_CUDA_TRY(cudaMemcpyAsync(&hc, counts, sizeof(int), cudaMemcpyDeviceToHost, st));
  NBK_CUDA_TRY(cudaStreamSynchronize(st));
  int64_t offs[2] = {0, hc};
  NBK_CUDA_TRY(cudaMemcpyAsync(d_off, offs, sizeof(offs), cudaMemcpyHostToDevice, st));
  int* found;
  double* fd2;
  NBK_TRY(alloc.get((void**)&found, sizeof(int) * (hc + 1)));
  NBK_TRY(alloc.get((void**)&fd2, sizeof(double) * (hc + 1)));
  a.offsets = d_off;
  a.out = found;
  a.outd2 = fd2;
  k_ball<true><<<1, 32 * kWpb, 0, st>>>(a); note_launch();
  k_mark<<<std::max(1, std::min(1024, (hc + 255) / 256)), 256, 0, st>>>(
      tv, target, fdist2, imark, found, fd2, d_off + 1, d_perm, d_mark, d_dist2,
      target_search); note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  NBK_CUDA_TRY(cudaStreamSynchronize(st));
  alloc.release_all_scratch(st);
  return NBK_OK;
}

}  // namespace nbk
