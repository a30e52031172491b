// Hand-written adjoint of the SPH density (no reference counterpart: the reference has
// no gradients). The forward pass is CalcDensity (KDCalcSmoothQuantities.cxx:203-305):
//   rho_i = sum_{j in N(i)} w_ij m_j + sum_{l : i in N(l)} w_li m_l,
//   w_ij  = 0.5 Wsm(q_ij) h_i^-3,  q_ij = r_ij / h_i,  h_i = 0.5 r_{i,K(i)}
// where K(i) is the farthest of the k neighbours and Wsm interpolates the kernel table.
// With the neighbour sets and each pair's table cell c frozen at the forward pass, Wsm is
// linear in q inside the cell: T(q) = T[c] + (T[c+1]-T[c]) (q - c delta) / delta, so
//   dw/dr = 0.5 h^-4 T'(q),   dw/dh = -0.5 h^-4 (3 T(q) + q T'(q)),   dh_i/dr_iK = 1/2.
// For L = sum_i w_i log rho_i, with g_i = w_i / rho_i and c_ij = g_i m_j + g_j m_i:
//   dL/dm_a = sum_{i: a in N(i)} g_i w_ia + sum_{j in N(a)} g_j w_aj
//   dL/dx_i += c_ij dw/dr (x_i - x_j)/r_ij   (and the opposite on x_j)
//   dL/dx_i += [sum_j c_ij dw/dh] (1/2) (x_i - x_K)/r_iK   (and the opposite on x_K).
// The backward kernel recomputes every weight from the saved neighbour lists (4 B per
// neighbour) instead of storing weights; one thread per particle, FP64 atomics for the
// contributions that land on other particles. What bounds it is the FP64 pipe: 30
// instructions a pair, 2.08 ms at 2^20, k = 32 (46 before the terms were rearranged, 3.45 ms). In the
// table coordinate u = q (kernres - 1) / 2 the line of a cell is T = A + D u and q T' = D u,
// factors of the particle alone (h^-3, h^-4, dL/drho_i) are taken out of the sums, the cell
// comes from the bits of u, and r and 1/r from one FP32 reciprocal square root (corrected in
// FP32 for r, by a cubic step for 1/r). Each pair's table cell is the forward pass's
// (int)(r / h * 0.5 * (kernres - 1)): from the fast u, and from the correctly rounded square
// root and division whenever u lies within 2^-30 of a cell edge (its own error is below
// 2^-40 there), so the frozen cells are exactly the forward's.
// Each saved row ends with the farthest neighbour, the one that set h_i.
#include <algorithm>

#include "nbk_build.h"

namespace nbk {

namespace {

// g_i = w_i / rho_i in place of w_i (tree order).
__global__ void k_adjoint_prep(double* wg, const double* __restrict__ rho, int64_t n) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) wg[i] = wg[i] / rho[i];
}

// r = sqrt(x) and 1 / r, both to about an ulp (0 < x inside FP32's range; see sqrt_newton).
__device__ __forceinline__ double root_pair(double x, double* inv) {
  const double r = sqrt_newton(x);
  const int hi = __double2hiint(x);
  if ((unsigned)(hi - ((1023 - 70) << 20)) > (unsigned)(170 << 20)) {
    *inv = 1.0 / r;
    return r;
  }
  float yf;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(yf) : "f"(f32_of_bits(hi, __double2loint(x))));
  const double y = f64_of_f32(yf), e = __fma_rn(-r, y, 1.0);
  *inv = __fma_rn(y, __fma_rn(e, e, e), y);
  return r;
}

__global__ void __launch_bounds__(128) k_adjoint(TreeView tv, int K, const int* __restrict__ nn,
                                                 const double* __restrict__ g,
                                                 const double* __restrict__ T, int kr,
                                                 double* gpos, double* gmass) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= tv.n) return;
  int ti = tv.pstart + i;
  const int* row = nn + (size_t)i * K;
  P4 xi = tv.pos[ti];
  const double gi = g[ti], mi = xi.m;
  // farthest neighbour: the one that set h_i in the forward pass (the row's last entry)
  const int kf = row[K - 1];
  if (kf < 0) return;  // too few neighbours, no row: reported by the search
  P4 xk = tv.pos[kf];
  const double best = dist2_exact(xi.x, xi.y, xi.z, xk.x, xk.y, xk.z);
  double irk;                                // 1 / r_iK
  const double hh = 0.5 * root_pair(best, &irk);  // the forward's h_i
  const double ih = 2.0 * irk;                // 1 / h_i
  const double norm = ih * ih * ih;
  const double hk = 0.5 * (double)(kr - 1), c1 = ih * hk;
  const double nh = -0.5 * norm * ih;  // dw/dh = nh (3 T + q T'), dw/dr = -nh T'
  const double pr = -nh * hk;          // dw/dr = pr D
  const double gn = 0.5 * gi * norm;
  const double* A = T + kr;
  const double* D = T + 3 * (size_t)kr;
  double acc = 0.0, gmi = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
  for (int s = 0; s < K; s++) {
    const int j = row[s];
    const P4 xj = tv.pos[j];
    const double dx = dsub(xi.x, xj.x), dy = dsub(xi.y, xj.y), dz = dsub(xi.z, xj.z);
    const double d2 = __fma_rn(dz, dz, __fma_rn(dy, dy, dmul(dx, dx)));
    double ir;  // 1 / r_ij (the target search excluded r = 0)
    const double u = dmul(root_pair(d2, &ir), c1);
    // the cell (int)u and the fraction of u in units of 2^-32, from its bits; the farthest
    // neighbour (the row's last) is at u = kernres - 1 exactly
    const int e = (__double2hiint(u) >> 20) - 1023;
    const unsigned long long m =
        ((unsigned long long)__double_as_longlong(u) << 11) | 0x8000000000000000ull;
    int c = e < 0 ? 0 : (int)(m >> (63 - min(e, 31)));
    const unsigned fr =
        (unsigned)((e < 0 ? m >> min(-1 - e, 63) : m << min(e + 1, 63)) >> 32);
    if (s == K - 1) {
      c = kr - 1;
    } else if (fr + 4u < 8u) {
      const double de = dist2_exact(xi.x, xi.y, xi.z, xj.x, xj.y, xj.z);
      c = (int)(dsqrt_call(de) / hh * 0.5 * (double)(kr - 1));
    }
    c = c < kr - 1 ? c : kr - 1;
    const double Dc = D[c];                    // 0 for the last entry
    const double t = dmul(Dc, u);              // q T'
    const double Tq = c < kr - 1 ? dadd(A[c], t) : T[kr - 1];
    const double gj = g[j];
    const double cij = __fma_rn(gj, mi, dmul(gi, xj.m));
    atomicAdd(&gmass[j], dmul(gn, Tq));
    gmi = __fma_rn(gj, Tq, gmi);
    acc = __fma_rn(cij, __fma_rn(3.0, Tq, t), acc);
    const double c0 = dmul(dmul(cij, ir), Dc);
    gx = __fma_rn(c0, dx, gx);
    gy = __fma_rn(c0, dy, gy);
    gz = __fma_rn(c0, dz, gz);
    const double cs = -dmul(c0, pr);
    atomicAdd(&gpos[3 * (size_t)j + 0], dmul(cs, dx));
    atomicAdd(&gpos[3 * (size_t)j + 1], dmul(cs, dy));
    atomicAdd(&gpos[3 * (size_t)j + 2], dmul(cs, dz));
  }
  const double ch = acc * nh * 0.5 * irk;
  double kx = ch * (xi.x - xk.x), ky = ch * (xi.y - xk.y), kz = ch * (xi.z - xk.z);
  atomicAdd(&gpos[3 * (size_t)kf + 0], -kx);
  atomicAdd(&gpos[3 * (size_t)kf + 1], -ky);
  atomicAdd(&gpos[3 * (size_t)kf + 2], -kz);
  atomicAdd(&gpos[3 * (size_t)ti + 0], __fma_rn(pr, gx, kx));
  atomicAdd(&gpos[3 * (size_t)ti + 1], __fma_rn(pr, gy, ky));
  atomicAdd(&gpos[3 * (size_t)ti + 2], __fma_rn(pr, gz, kz));
  atomicAdd(&gmass[ti], gmi * 0.5 * norm);
}

}  // namespace

int run_density_adjoint(const TreeView& tv, int k, const int* d_nn, double* d_w_tree,
                        const double* d_rho_tree, const double* kernel, int kernres,
                        double* d_gpos_tree, double* d_gmass_tree, cudaStream_t st) {
  if (tv.n == 0) return NBK_OK;
  NBK_CUDA_TRY(cudaMemsetAsync(d_gpos_tree, 0, sizeof(double) * 3 * tv.n, st));
  NBK_CUDA_TRY(cudaMemsetAsync(d_gmass_tree, 0, sizeof(double) * tv.n, st));
  Phase ph("adjoint_backward", st);
  k_adjoint_prep<<<(unsigned)(((int64_t)tv.n + 255) / 256), 256, 0, st>>>(d_w_tree, d_rho_tree,
                                                                          tv.n);
  note_launch();
  k_adjoint<<<(tv.n + 127) / 128, 128, 0, st>>>(tv, k, d_nn, d_w_tree, kernel, kernres,
                                                d_gpos_tree, d_gmass_tree);
  note_launch();
  NBK_CUDA_TRY(cudaGetLastError());
  return NBK_OK;
}

}  // namespace nbk
