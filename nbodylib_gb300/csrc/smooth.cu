// SPH smoothing over the Nsmooth nearest neighbours (KDCalcSmoothQuantities.cxx):
//   CalcSmoothVel, CalcSmoothVelDisp, CalcSmoothVelSkew, CalcSmoothVelKurtosis (:480-766),
//   symmetric sums over every particle's neighbours, scattered to both ends of each pair;
//   CalcVelDensityWithPhysDensity[Particle] (:393-478, :922-990);
//   CalcSmoothVel/CalcSmoothVelDisp {Particle,Position} (:992-1091, :1209-1306) and
//   CalcSmoothLocalMean/CalcSmoothLocalDisp {Particle,Position} (:1539-1700), one-sided.
//
// The neighbours come from the kNN search (the group search for every particle, a warp per
// query else) as rows of indices with the farthest last; a thread per query then runs over
// its row. What belongs to a particle and not to a pair is prepared once per particle in
// tree order (m / rho, the mean velocity, the inverse powers of the dispersion: divisions
// and permutations out of the pair loop), and the every-particle sums are gathered with FP64
// atomics in tree order, where neighbours are close in memory, then permuted. The summation
// order (not the terms) differs from the reference's. A row costs 4 B per neighbour each way;
// trees of more than kSliceMax particles go slice by slice, so that the rows stay small.
//
// What bounds it: the search, and in k_smooth_rows the FP64 pipe (85% busy), 18 instructions a
// pair for CalcSmoothVel and 36 for CalcSmoothVelDisp (its nine sums are six, the matrix being
// symmetric). As epilogues of a lane-per-query search with all divisions per pair the two took
// 8.2 ms each at 2^20 clustered particles, Nsmooth = 32; now the searches take 2.65 ms
// each and everything after them 3.8 ms for the two.
#include <algorithm>

#include "knn_wq.cuh"

namespace nbk {

namespace {

constexpr int64_t kSliceMax = int64_t(1) << 23;  // queries per slice of rows

// One particle's share of the pair terms, tree order.
struct SmoothPrep {
  const double* mr;  // m / rho
  const V4* sv;      // mean velocity (moment forms)
  const V4* iv;      // inverse power of the dispersion's diagonal (skewness, kurtosis)
  const double* wt;  // weights (local mean and dispersion)
};

__global__ void k_smooth_prep(SmoothArgs s, int n, int which, double* mr, V4* sv, V4* iv,
                              double* wt) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t id = s.k.tv.perm[t];
  mr[t] = s.k.tv.pos[t].m / s.rho[id];
  if (sv) sv[t] = make_v4(s.smvel[3 * id], s.smvel[3 * id + 1], s.smvel[3 * id + 2], 0.0);
  if (iv) {
    double v[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const double d = s.disp[9 * id + 4 * k];
      // the reference's 1 / pow(d, 1.5), and 1 / (d d)
      v[k] = which == kSmVelSkew ? 1.0 / dmul(d, __dsqrt_rn(d)) : 1.0 / dmul(d, d);
    }
    iv[t] = make_v4(v[0], v[1], v[2], 0.0);
  }
  if (wt) wt[t] = s.weight[id];
}

// Sums per particle in tree order to input order; the dispersion's six to its nine.
template <int W>
__global__ void k_smooth_out(const double* acc, const int* perm, double* out, int n) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int64_t id = perm[t];
  if (W == 6) {
    const int at[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma unroll
    for (int c = 0; c < 9; c++) out[9 * id + c] = acc[6 * (int64_t)t + at[c]];
  } else {
#pragma unroll
    for (int c = 0; c < W; c++) out[W * id + c] = acc[W * (int64_t)t + c];
  }
}

template <int SM>
__global__ void __launch_bounds__(128) k_smooth_rows(SmoothArgs s, SmoothPrep P, int K,
                                                     double* acc_out) {
  const KnnArgs& a = s.k;
  const TreeView& tv = a.tv;
  const int qi = blockIdx.x * blockDim.x + threadIdx.x;
  if (qi >= a.nq) return;
  const int* row = a.nn + (size_t)qi * K;
  constexpr bool kSym = SM == kSmVel || SM == kSmVelDisp || SM == kSmVelSkew || SM == kSmVelKurt;
  int self = -1;
  double x, y, z;
  if (a.qmode == 1) {
    x = a.qx[3 * (size_t)qi];
    y = a.qx[3 * (size_t)qi + 1];
    z = a.qx[3 * (size_t)qi + 2];
  } else {
    self = a.qmode == 0 ? a.q0 + qi : a.qidx[qi];
    if (self < 0 || self >= tv.n) return;  // reported by the search
    const P4 p = tv.pos[self];
    x = p.x;
    y = p.y;
    z = p.z;
  }
  if (row[K - 1] < 0) return;  // too few neighbours: reported by the search
  const int kr = a.kernres;
  const double* T = a.kernel;
  // the weights of the neighbours: h = half the largest distance
  double top;
  {
    const P4 c = tv.pos[row[K - 1]];
    const double dx = dsub(x, c.x), dy = dsub(y, c.y), dz = dsub(z, c.z);
    top = __fma_rn(dz, dz, __fma_rn(dy, dy, dmul(dx, dx)));
  }
  const double ih = two_rsqrt(top), c1 = dmul(ih, 0.5 * (double)(kr - 1));
  const double norm = dmul(dmul(ih, ih), ih);
  const double wnorm = kSym ? 0.5 * norm : norm;  // the symmetric forms carry the 1/2
  V4 vi = make_v4(0, 0, 0, 0), si = vi;
  double wi = 0.0;  // this particle's factor in its neighbours' sums
  if (kSym) {
    vi = tv.vel[self];
    wi = dmul(wnorm, P.mr[self]);
    if (SM != kSmVel) si = P.sv[self];
  }
  V4 ivi = make_v4(0, 0, 0, 0);
  if (SM == kSmVelSkew || SM == kSmVelKurt) ivi = P.iv[self];
  if (SM == kSmVelDispOne)
    si = make_v4(s.smvel[3 * (size_t)qi], s.smvel[3 * (size_t)qi + 1], s.smvel[3 * (size_t)qi + 2],
                 0.0);
  const double mean = SM == kSmDispOne ? s.mean[qi] : 0.0;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (int q = 0; q < K; q++) {
    const int j = row[q];
    const P4 c = tv.pos[j];
    const double dx = dsub(x, c.x), dy = dsub(y, c.y), dz = dsub(z, c.z);
    const double d2 = __fma_rn(dz, dz, __fma_rn(dy, dy, dmul(dx, dx)));
    // the farthest neighbour sits at q = 2 exactly: the table's last entry
    // (compared by their bits: FP64 compares take the FP64 pipe)
    const double w = dkey(d2) == dkey(top) ? T[kr - 1] : w_at_u(dmul(sqrt_newton(d2), c1), kr, T);
    // W_ij m_j / rho_j into the query (times wnorm: at the end, but for the kurtosis, whose
    // terms are shifted), W_ij m_i / rho_i into neighbour j
    const double ta = dmul(SM == kSmVelKurt ? dmul(w, wnorm) : w, P.mr[j]);
    const double tb = dmul(w, wi);
    if (SM == kSmMeanOne) {
      acc[0] = __fma_rn(ta, P.wt[j], acc[0]);
    } else if (SM == kSmDispOne) {
      const double dl = dsub(P.wt[j], mean);
      acc[0] = __fma_rn(dmul(ta, dl), dl, acc[0]);
    } else if (SM == kSmVel || SM == kSmVelOne) {
      const V4 vj = tv.vel[j];
      acc[0] = __fma_rn(ta, vj.x, acc[0]);
      acc[1] = __fma_rn(ta, vj.y, acc[1]);
      acc[2] = __fma_rn(ta, vj.z, acc[2]);
      if (SM == kSmVel) {
        double* o = acc_out + 3 * (size_t)j;
        atomicAdd(o, dmul(tb, vi.x));
        atomicAdd(o + 1, dmul(tb, vi.y));
        atomicAdd(o + 2, dmul(tb, vi.z));
      }
    } else {
      const V4 vj = tv.vel[j];
      const double d[3] = {dsub(vj.x, si.x), dsub(vj.y, si.y), dsub(vj.z, si.z)};
      if (SM == kSmVelDisp || SM == kSmVelDispOne) {
        const double e[3] = {dmul(ta, d[0]), dmul(ta, d[1]), dmul(ta, d[2])};
        acc[0] = __fma_rn(e[0], d[0], acc[0]);
        acc[1] = __fma_rn(e[0], d[1], acc[1]);
        acc[2] = __fma_rn(e[0], d[2], acc[2]);
        acc[3] = __fma_rn(e[1], d[1], acc[3]);
        acc[4] = __fma_rn(e[1], d[2], acc[4]);
        acc[5] = __fma_rn(e[2], d[2], acc[5]);
      }
      if (kSym) {
        const V4 sj = P.sv[j];
        const double u[3] = {dsub(vi.x, sj.x), dsub(vi.y, sj.y), dsub(vi.z, sj.z)};
        if (SM == kSmVelDisp) {
          const double f[3] = {dmul(tb, u[0]), dmul(tb, u[1]), dmul(tb, u[2])};
          double* o = acc_out + 6 * (size_t)j;
          atomicAdd(o, dmul(f[0], u[0]));
          atomicAdd(o + 1, dmul(f[0], u[1]));
          atomicAdd(o + 2, dmul(f[0], u[2]));
          atomicAdd(o + 3, dmul(f[1], u[1]));
          atomicAdd(o + 4, dmul(f[1], u[2]));
          atomicAdd(o + 5, dmul(f[2], u[2]));
        } else {
          const V4 ivj = P.iv[j];
          const double ii[3] = {ivi.x, ivi.y, ivi.z}, ij[3] = {ivj.x, ivj.y, ivj.z};
          double* o = acc_out + 3 * (size_t)j;
#pragma unroll
          for (int k = 0; k < 3; k++) {
            const double a3 = dmul(dmul(dmul(ta, d[k]), d[k]), d[k]);
            const double b3 = dmul(dmul(dmul(tb, u[k]), u[k]), u[k]);
            if (SM == kSmVelSkew) {
              acc[k] = __fma_rn(a3, ii[k], acc[k]);
              atomicAdd(o + k, dmul(b3, ij[k]));
            } else {
              // the reference subtracts 3 in every neighbour's term
              acc[k] = dadd(acc[k], dsub(dmul(dmul(a3, d[k]), ii[k]), 3.0));
              atomicAdd(o + k, dsub(dmul(dmul(b3, u[k]), ij[k]), 3.0));
            }
          }
        }
      }
    }
  }
  if (SM != kSmVelKurt)
#pragma unroll
    for (int k = 0; k < 6; k++) acc[k] = dmul(acc[k], wnorm);
  constexpr int kAcc = SM == kSmVelDisp || SM == kSmVelDispOne ? 6
                       : SM == kSmMeanOne || SM == kSmDispOne  ? 1
                                                               : 3;
  if (kSym) {
#pragma unroll
    for (int k = 0; k < kAcc; k++) atomicAdd(acc_out + kAcc * (size_t)self + k, acc[k]);
  } else if (SM == kSmVelDispOne) {
    const int at[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
#pragma unroll
    for (int c = 0; c < 9; c++) s.out[9 * (size_t)qi + c] = acc[at[c]];
  } else {
#pragma unroll
    for (int k = 0; k < kAcc; k++) s.out[kAcc * (size_t)qi + k] = acc[k];
  }
}

// CalcVelDensityWithPhysDensity: a warp per query, a neighbour per lane and slot. |dv| of the
// Nsearch neighbours, the Nsmooth smallest kept (as CalcVelDensity); the physical h is half
// the largest *squared* distance, as the reference computes it (:428); a table index past the
// end gives the table's last entry (the reference reads past its table there).
template <int S>
__global__ void __launch_bounds__(256) k_smooth_velphys(SmoothArgs s, SmoothPrep P, int K) {
  const unsigned FULL = 0xffffffffu;
  const KnnArgs& a = s.k;
  const TreeView& tv = a.tv;
  const int lane = threadIdx.x & 31;
  const int qi = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (qi >= a.nq) return;
  const int self = a.qmode == 0 ? a.q0 + qi : a.qidx[qi];
  if (self < 0 || self >= tv.n) return;  // reported by the search
  const int kr = a.kernres;
  const double* T = a.kernel;
  const int* row = a.nn + (size_t)qi * K;
  if (row[K - 1] < 0) return;  // too few neighbours: reported by the search
  const P4 x = tv.pos[self];
  const V4 v = tv.vel[self];
  double d2[S];
  long long vk[S], top = 0;
#pragma unroll
  for (int q = 0; q < S; q++) {
    const int p = q * 32 + lane;
    vk[q] = kWqSent;
    d2[q] = 0.0;
    if (p < K) {
      const int j = row[p];
      const V4 vj = tv.vel[j];
      const P4 c = tv.pos[j];
      vk[q] = dkey(sqrt_newton(dist2_exact(v.x, v.y, v.z, vj.x, vj.y, vj.z)));
      d2[q] = dist2_exact(x.x, x.y, x.z, c.x, c.y, c.z);
      top = max(top, dkey(d2[q]));
    }
  }
  const int ns = min(s.nsmooth, K);
  int rk[S];
  if (ns < K) wq_ranks<S>(vk, lane, K, rk);
  bool sel[S];
  long long vmax = 0;
#pragma unroll
  for (int q = 0; q < S; q++) {
    sel[q] = q * 32 + lane < K && (ns == K || rk[q] < ns);
    if (sel[q]) vmax = max(vmax, vk[q]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vmax = max(vmax, __shfl_xor_sync(FULL, vmax, o));
    top = max(top, __shfl_xor_sync(FULL, top, o));
  }
  const double vih = recip_newton(0.5 * __longlong_as_double(vmax));
  const double vnorm = dmul(dmul(vih, vih), vih);
  const double ih = recip_newton(0.5 * __longlong_as_double(top));
  const double norm = dmul(dmul(ih, ih), ih);
  const double hk = 0.5 * (double)(kr - 1), mr = P.mr[self];
  double acc = 0.0;
#pragma unroll
  for (int q = 0; q < S; q++) {
    if (!sel[q]) continue;
    const double vw = vk[q] == vmax  // the largest |dv| is at q = 2 exactly
                          ? T[kr - 1]
                          : w_at_u(dmul(dmul(__longlong_as_double(vk[q]), vih), hk), kr, T);
    const double w = w_at_u(dmul(dmul(sqrt_newton(d2[q]), ih), hk), kr, T);
    acc = __fma_rn(dmul(vw, vnorm), dmul(dmul(w, norm), mr), acc);
  }
  acc = warp_sum(acc);
  if (lane == 0) s.out[a.qmode == 0 ? tv.perm[self] : qi] = acc;
}

// Start and size of the slice-th of the 2^levels nodes of a level (KDTree.cxx:1012).
void slice_range(int64_t n, int levels, int slice, int64_t* start, int64_t* size) {
  int64_t s = 0;
  for (int i = levels - 1; i >= 0; i--) {
    const int64_t l = (n - 1) / 2 + 1;
    if ((slice >> i) & 1) {
      s += l;
      n -= l;
    } else {
      n = l;
    }
  }
  *start = s;
  *size = n;
}

template <int SM>
int rows_pass(const SmoothArgs& s, const SmoothPrep& P, int K, double* acc, cudaStream_t st) {
  k_smooth_rows<SM><<<(unsigned)((s.k.nq + 127) / 128), 128, 0, st>>>(s, P, K, acc);
  note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  return NBK_OK;
}

}  // namespace

int launch_smooth(const SmoothArgs& s0, int which, DevAlloc& alloc, cudaStream_t st) {
  const int K = s0.k.kheap;
  if (which < kSmVel || which > kSmDispOne) {
    set_error("unknown smoothing quantity");
    return NBK_ERR_INVALID;
  }
  if (K > 128) {
    set_error("smoothing over more than 128 neighbours is not supported");
    return NBK_ERR_UNSUPPORTED;
  }
  if (s0.k.nq == 0) return NBK_OK;
  const int n = s0.k.tv.n;
  const int64_t nq = s0.k.nq;
  const bool sym = which <= kSmVelKurt, every = s0.k.qmode == 0;
  const int width = which == kSmVelDisp ? 6 : 3;
  // slices of the queries: nodes of one level for every particle, plain ranges else
  int levels = 0;
  while (every && (nq >> levels) > kSliceMax) levels++;
  const int64_t step = every ? (((nq - 1) >> levels) + 1) : std::min(nq, kSliceMax);
  const int slices = every ? 1 << levels : (int)((nq + step - 1) / step);
  double *mr, *acc = nullptr, *wt = nullptr;
  V4 *sv = nullptr, *iv = nullptr;
  int *rows, *fb = nullptr;
  std::vector<DevPart> parts{{(void**)&mr, sizeof(double) * n},
                             {(void**)&rows, sizeof(int) * step * K}};
  if (sym) parts.push_back({(void**)&acc, sizeof(double) * width * n});
  if (sym && which != kSmVel) parts.push_back({(void**)&sv, sizeof(V4) * n});
  if (which == kSmVelSkew || which == kSmVelKurt) parts.push_back({(void**)&iv, sizeof(V4) * n});
  if (which == kSmMeanOne || which == kSmDispOne) parts.push_back({(void**)&wt, sizeof(double) * n});
  if (every) parts.push_back({(void**)&fb, sizeof(int) * (step + 1)});
  if (s0.k.qmode == 1) parts.push_back({(void**)&fb, sizeof(int) * (step / 16 + 5)});
  NBK_TRY(alloc.get_block(parts));
  if (sym) NBK_CUDA_TRY(cudaMemsetAsync(acc, 0, sizeof(double) * width * n, st));
  Phase ph("smooth", st);
  const unsigned nb = (unsigned)((n + 255) / 256);
  k_smooth_prep<<<nb, 256, 0, st>>>(s0, n, which, mr, sv, iv, wt);
  note_launch();
  const SmoothPrep P{mr, sv, iv, wt};
  for (int i = 0; i < slices; i++) {
    SmoothArgs s = s0;
    s.k.nn = rows;
    s.k.fb = fb;
    if (every) {
      int64_t start, size;
      slice_range(nq, levels, i, &start, &size);
      s.k.q0 = (int)start;
      s.k.nq = (int)size;
      s.k.slices = levels;
      s.k.slice = i;
    } else {
      const int64_t o = i * step;
      s.k.nq = (int)std::min(step, nq - o);
      if (s.k.qidx) s.k.qidx += o;
      if (s.k.qx) s.k.qx += 3 * o;
      if (s.smvel) s.smvel += 3 * o;
      if (s.mean) s.mean += o;
      s.out += o * (which == kSmVelDispOne ? 9 : which == kSmVelOne ? 3 : 1);
    }
    NBK_TRY(launch_knn(s.k, kEpiSave, st));
    switch (which) {
      case kSmVel: NBK_TRY(rows_pass<kSmVel>(s, P, K, acc, st)); break;
      case kSmVelDisp: NBK_TRY(rows_pass<kSmVelDisp>(s, P, K, acc, st)); break;
      case kSmVelSkew: NBK_TRY(rows_pass<kSmVelSkew>(s, P, K, acc, st)); break;
      case kSmVelKurt: NBK_TRY(rows_pass<kSmVelKurt>(s, P, K, acc, st)); break;
      case kSmVelOne: NBK_TRY(rows_pass<kSmVelOne>(s, P, K, acc, st)); break;
      case kSmVelDispOne: NBK_TRY(rows_pass<kSmVelDispOne>(s, P, K, acc, st)); break;
      case kSmMeanOne: NBK_TRY(rows_pass<kSmMeanOne>(s, P, K, acc, st)); break;
      case kSmDispOne: NBK_TRY(rows_pass<kSmDispOne>(s, P, K, acc, st)); break;
      default: {
        const unsigned blocks = (unsigned)((s.k.nq + 7) / 8);
        if (K <= 32) k_smooth_velphys<1><<<blocks, 256, 0, st>>>(s, P, K);
        else if (K <= 64) k_smooth_velphys<2><<<blocks, 256, 0, st>>>(s, P, K);
        else k_smooth_velphys<4><<<blocks, 256, 0, st>>>(s, P, K);
        note_launch();
        NBK_CUDA_TRY(cudaGetLastError());
      }
    }
  }
  if (sym) {
    if (width == 6) k_smooth_out<6><<<nb, 256, 0, st>>>(acc, s0.k.tv.perm, s0.out, n);
    else k_smooth_out<3><<<nb, 256, 0, st>>>(acc, s0.k.tv.perm, s0.out, n);
    note_launch();
    NBK_CUDA_TRY(cudaGetLastError());
  }
  return NBK_OK;
}

}  // namespace nbk
