// Quasi-static Newton / CG (sm_100a), FP64.
//
// Replaces Peridigm::executeQuasiStatic (src/core/Peridigm.cpp:2470-3043) with
// its residual (computeQuasiStaticResidual, :4176-4317), tangent
// (ElasticMaterial::computeAutomaticDifferentiationJacobian,
// src/materials/Peridigm_ElasticMaterial.cpp:258-383, Scale(-1) at
// Peridigm.cpp:2800) and Belos CG (:2551-2573, :3321-3362):
//  * residual r = V (f_int + f_ext), rows of prescribed dofs zeroed;
//  * tangent K = -d r / d u applied matrix-free: the exact linearization of
//    the LPS force in two bond passes (d theta, then d f) over per-bond
//    geometry built once per state (unit deformed bond, V_j om zeta,
//    V_j T/|Y|, V_j om (alpha_i + alpha_j)), rows and columns of prescribed
//    dofs replaced by identity (applyKinematicBC_InsertZerosAndSetDiagonal);
//  * preconditioned CG with deterministic FP64 dot products; block-Jacobi
//    preconditioner = inverses of the analytic 3x3 diagonal blocks of K
//    (the reference's "Block 3x3" preconditioner, Peridigm.cpp:1603-1646);
//    the two-level and learned preconditioners add k_coarse.cu's coarse
//    correction and k_mpnn.cu's learned middle level to it;
//  * Newton with a backtracking step on the reference's convergence metric
//    ||r||_2 + 20 ||r||_inf (Peridigm.cpp:4316).
// For a bond (i,j) with Y = y_j - y_i, e = |Y| - |X|, de = Yhat.(w_j - w_i):
//   d theta_i = sum 3 omega zeta de V_j / m_i
//   t_ij = omega (zeta theta_i q_i + alpha_i e),  q = 3K/m - alpha/3, alpha = 15mu/m
//   dt_ij = omega (zeta dtheta_i q_i + alpha_i de)
//   d f_i = sum V_j [ (dt_ij + dt_ji) Yhat + (t_ij + t_ji) (dw - Yhat de)/|Y| ]
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "cg.cuh"
#include "grid_sync.cuh"
#include "pd_internal.cuh"

namespace pdb {

constexpr int kQsBlock = 256;
constexpr int kQsTpo = 8;
// Bonds per lane in flight in the tangent passes and their resident blocks per
// SM, at 60x60x60 points (24.9 M bonds): first pass 126 us at 4 bonds and 5
// blocks (48 registers; 6 blocks 128, unbounded 132 to 167), second 200 us at
// 4 bonds and 4 blocks (64 registers; 2 bonds 203, 3 blocks 229, 5 blocks 247).
#ifndef PD_QS_BATCH
#define PD_QS_BATCH 4
#endif
#ifndef PD_QS_BATCH2
#define PD_QS_BATCH2 4
#endif
#ifndef PD_QS_MINB
#define PD_QS_MINB 5
#endif
#ifndef PD_QS_MINB2
#define PD_QS_MINB2 4
#endif
constexpr int kQsBatch = PD_QS_BATCH, kQsBatch2 = PD_QS_BATCH2;
#ifndef PD_QS_WIDE
#define PD_QS_WIDE 4096
#endif
// Bodies up to this size take 32 lanes per point in the tangent passes, larger
// ones 8. Both passes of one product, us, cubes of points at 32 and 8 lanes:
// 14^3 12.8 and 15.1, 16^3 13.7 and 15.2, 17^3 16.3 and 15.6, 20^3 22.4 and
// 17.1, 25^3 37.2 and 22.7, 40^3 174 and 116: few points leave lanes idle, more
// of them pay for the wider sums and the rows' idle last lanes.
constexpr int64_t kQsWide = PD_QS_WIDE;
constexpr int kRedBlocks = 296;  // 2 x 148 SMs: fixed, so reductions are deterministic

struct QsState {
  DBuf<double4> yq;    // coordinates x + u + du
  DBuf<double4> abq;   // (theta, q, alpha, q/m)
  DBuf<double4> w;     // CG direction (p, dtheta)
  DBuf<double> th, nd, f, r, du, x, z, q, pred, dinv, partial, scal;
  DBuf<uint8_t> fixed;  // bit c: dof c prescribed
  int64_t n = 0;
  bool coarse_on = false;  // the preconditioner adds the aggregate coarse correction (k_coarse.cu)
  // Per-bond tangent geometry at the current (y, theta, q, alpha), rebuilt
  // after every change of the state (geo_dirty), see k_qs_bond_geom; zero for
  // broken bonds.
  DBuf<double4> geo;
  DBuf<double2> gco;
  bool geo_dirty = true;
  // Coarse-operator reuse: the operator is rebuilt when the model changed, or
  // when a solve needs more than 1.3x (+5) the CG iterations of the first solve
  // after the last rebuild (the tangent drifted from the one it was built at).
  double coarse_cell = -1.0;
  int64_t coarse_ref_iters = -1;
  bool coarse_rebuild = true;
  // The operator the CG products and block-Jacobi blocks use: jm rho I + jk K
  // (quasi-static: K; implicit dynamics: rho I + beta dt^2 K).
  double jk = 1.0, jm = 0.0;
  DBuf<double> v2;  // implicit dynamics: velocity predictor
  DBuf<double> cg_b, cg_x0;  // learned-preconditioner CG: right-hand side and restart point (kept, not reallocated)
  DBuf<CgCtl> ctl;           // scalars and state of the running solve
  CgReport* report = nullptr;      // its progress, in a mapped page (made by the first solve that reports)
  CgReport* report_dev = nullptr;
  bool no_report = false;          // (not to be had)
  // one-launch solve: threads per block (-1: not determined, 0: the general
  // loop) and bonds per lane, for rows of up to small_max_row bonds
  int small_threads = -1, small_slots = 0, small_max_row = -1;
  ~QsState() {
    if (report) {
      cudaHostUnregister(report);
      free(report);
    }
  }
};

__device__ __forceinline__ double qs_omega(int kind, double zeta, double h) {
  if (kind == PD_INFLUENCE_ONE) return 1.0;
  if (kind == PD_INFLUENCE_PARABOLIC_DECAY) {
    if (zeta > h) return 0.0;
    const double s = zeta / h;
    return s < 0.5 ? 1.0 : -4.0 * s * s + 4.0 * s;
  }
  return exp(-(zeta * zeta) / (h * h * 0.16));
}

template <int TPO = kQsTpo, typename T>
__device__ __forceinline__ T qs_group_sum(T v) {
#pragma unroll
  for (int o = TPO / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// y = (x + u) + du (Peridigm.cpp:2684-2687 operation order)
__global__ void k_qs_positions(int64_t n, const double4* __restrict__ xv, const double* __restrict__ u,
                               const double* __restrict__ du, double4* __restrict__ y) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double4 x = xv[i];
  y[i] = make_double4((x.x + u[3 * i]) + du[3 * i], (x.y + u[3 * i + 1]) + du[3 * i + 1],
                      (x.z + u[3 * i + 2]) + du[3 * i + 2], 0.0);
}

// abq.w = q/m for the block-diagonal term
__global__ void k_qs_qm(int64_t n, const double4* __restrict__ pt, double4* __restrict__ ab) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ab[i].w = ab[i].y / pt[i].x;
}

// r = V f with prescribed rows zeroed; block partials of sum r^2 and max |r|.
__global__ void k_qs_residual(int64_t n, const double* __restrict__ f, const double4* __restrict__ xv,
                              const uint8_t* __restrict__ fixed, double* __restrict__ r,
                              double* __restrict__ partial) {
  __shared__ double s2[kQsBlock], sm[kQsBlock];
  double a2 = 0.0, am = 0.0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < 3 * n; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = k / 3;
    const int c = (int)(k - 3 * i);
    double v = f[k] * xv[i].w;
    if ((fixed[i] >> c) & 1) v = 0.0;
    r[k] = v;
    a2 += v * v;
    am = fmax(am, fabs(v));
  }
  s2[threadIdx.x] = a2;
  sm[threadIdx.x] = am;
  __syncthreads();
  for (int o = kQsBlock / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      s2[threadIdx.x] += s2[threadIdx.x + o];
      sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = s2[0];
    partial[2 * blockIdx.x + 1] = sm[0];
  }
}

// Sums (even slots) and maxima (odd slots) of kRedBlocks partial pairs, or
// plain sums of `width` interleaved partials; fixed order.
__global__ void k_qs_reduce(const double* __restrict__ partial, int nblk, int width, int mode,
                            double* __restrict__ out) {
  __shared__ double s[kQsBlock];
  for (int c = 0; c < width; ++c) {
    double a = 0.0;
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
      const double v = partial[width * b + c];
      a = (mode == 1 && c == 1) ? fmax(a, v) : a + v;
    }
    s[threadIdx.x] = a;
    __syncthreads();
    for (int o = kQsBlock / 2; o > 0; o >>= 1) {
      if (threadIdx.x < o) s[threadIdx.x] = (mode == 1 && c == 1) ? fmax(s[threadIdx.x], s[threadIdx.x + o])
                                                                   : s[threadIdx.x] + s[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) out[c] = s[0];
    __syncthreads();
  }
}

// Per-bond tangent geometry (one lane group per owner, bonds strided over
// lanes). With c1 = V_j om zeta and yh = Y/|Y| the terms of the two passes are
//   c1 yh.dw                           = G.dw                       G = c1 yh
//   V_j [dT yh + (T/|Y|) (dw - yh de)] = (q dth_i + q dth_j + k2 (G.dw)) G + cx dw
//   cx = V_j T/|Y|, k2 = (V_j om (alpha_i + alpha_j) - cx) / c1^2
// The neighbor's id rides in the fourth number of G's record: the first pass of
// a CG iteration streams 32 B per bond and the second 48, a record in one
// 256-bit load. (yh, c1, the two coefficients and the id apart were 36 and 52 B
// in twice as many loads; G in three planes, 28 and 44 B, took more L1
// wavefronts than the bytes it saved; gathering the coordinates instead of
// streaming G, 12 and 28 B, left both passes bound by the L1's gathers.) A bond of c1 = 0 (coincident points) takes c1 = 1e-100: no
// term in the first pass, its own in the second.
__global__ void __launch_bounds__(kQsBlock) k_qs_bond_geom(int64_t n, const int64_t* __restrict__ row,
                                                           const int32_t* __restrict__ col,
                                                           const uint8_t* __restrict__ dmg,
                                                           const double4* __restrict__ xv,
                                                           const double4* __restrict__ y,
                                                           const double4* __restrict__ ab,
                                                           const double* __restrict__ hp, int influence,
                                                           double4* __restrict__ g,
                                                           double2* __restrict__ gc) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kQsTpo;
  const int lane = threadIdx.x & (kQsTpo - 1);
  if (i >= n) return;
  const double4 xi = xv[i], yi = y[i], ai = ab[i];
  const double h = hp[i];
  for (int64_t b = row[i] + lane; b < row[i + 1]; b += kQsTpo) {
    if (dmg[b]) {
      g[b] = make_double4(0.0, 0.0, 0.0, __longlong_as_double(col[b]));
      gc[b] = make_double2(0.0, 0.0);
      continue;
    }
    const int32_t j = col[b];
    const double4 xj = xv[j], yj = y[j], aj = ab[j];
    const double X0 = xj.x - xi.x, X1 = xj.y - xi.y, X2 = xj.z - xi.z;
    const double Y0 = yj.x - yi.x, Y1 = yj.y - yi.y, Y2 = yj.z - yi.z;
    const double zeta = sqrt(X0 * X0 + X1 * X1 + X2 * X2);
    const double dY = sqrt(Y0 * Y0 + Y1 * Y1 + Y2 * Y2);
    const double e = dY - zeta;
    const double om = qs_omega(influence, zeta, h);
    const double T = om * (zeta * (ai.x * ai.y + aj.x * aj.y) + (ai.z + aj.z) * e);
    const double V = xj.w;
    const double cx = V * T / dY, cd = V * om * (ai.z + aj.z) - cx;
    double c1 = V * om * zeta;
    if (c1 == 0.0 && cd != 0.0) c1 = 1e-100;
    const double s = c1 / dY;
    g[b] = make_double4(s * Y0, s * Y1, s * Y2, __longlong_as_double(j));
    gc[b] = make_double2(c1 != 0.0 ? cd / c1 / c1 : 0.0, cx);
  }
}

// 256-bit loads: of a bond's record (read once per pass), of a point's (p, q dtheta).
__device__ __forceinline__ double4 ld_bond(const double4* p) {
  double4 r;
  asm("ld.global.cs.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
  return r;
}
__device__ __forceinline__ double4 ld_w(const double4* p) {
  double4 r;
  asm("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p));
  return r;
}
__device__ __forceinline__ int64_t bond_id(const double4& g) { return __double_as_longlong(g.w); }

// Tangent pass 1 on the geometry: w[i].w = q_i dtheta_i = 3 (q_i/m_i) sum_j G_ij.(w_j - w_i)
// (a solve that has ended makes the kernel return)
template <int TPO>
__global__ void __launch_bounds__(kQsBlock, PD_QS_MINB) k_qs_dtheta_g(int64_t n, const int64_t* __restrict__ row,
                                                          const double4* __restrict__ g,
                                                          const double4* __restrict__ ab,
                                                          const double4* __restrict__ pt, double4* w,
                                                          const CgCtl* __restrict__ ctl) {
  if (ctl->state) return;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / TPO;
  const int lane = threadIdx.x & (TPO - 1);
  const bool valid = i < n;
  double acc = 0.0;
  if (valid) {
    const double4 wi = w[i];
    const int64_t b1 = row[i + 1];
    int64_t b = row[i] + lane;
    auto bond = [&](const double4& gb, const double4& wj) {
      acc += gb.x * (wj.x - wi.x) + gb.y * (wj.y - wi.y) + gb.z * (wj.z - wi.z);
    };
    // batches of kQsBatch bonds per lane: stream loads, then gathers, then the
    // sums in bond order (the same order as one bond at a time)
    for (; b + (kQsBatch - 1) * TPO < b1; b += kQsBatch * TPO) {
      double4 gb[kQsBatch], wj[kQsBatch];
#pragma unroll
      for (int k = 0; k < kQsBatch; ++k) gb[k] = ld_bond(g + b + k * TPO);
#pragma unroll
      for (int k = 0; k < kQsBatch; ++k) wj[k] = ld_w(w + bond_id(gb[k]));
#pragma unroll
      for (int k = 0; k < kQsBatch; ++k) bond(gb[k], wj[k]);
    }
    for (; b < b1; b += TPO) {
      const double4 gb = ld_bond(g + b);
      bond(gb, ld_w(w + bond_id(gb)));
    }
  }
  acc = qs_group_sum<TPO>(acc);
  if (valid && lane == 0) w[i].w = 3.0 * (ab[i].y / pt[i].x) * acc;
}

// Tangent pass 2 on the geometry: q = K p = -V d f (prescribed rows: q = p), or
// (jm rho I + jk K) p for implicit dynamics; p.q goes to ctl->pq
template <int TPO>
__global__ void __launch_bounds__(kQsBlock, PD_QS_MINB2) k_qs_df_g(int64_t n, const int64_t* __restrict__ row,
                                                      const double4* __restrict__ g,
                                                      const double2* __restrict__ gc,
                                                      const double4* __restrict__ xv,
                                                      const double4* __restrict__ w,
                                                      const uint8_t* __restrict__ fixed, double* __restrict__ q,
                                                      double* __restrict__ partial, const double4* __restrict__ pt,
                                                      double jk, double jm, CgCtl* __restrict__ ctl) {
  if (ctl->state) return;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / TPO;
  const int lane = threadIdx.x & (TPO - 1);
  const bool valid = i < n;
  double d0 = 0.0, d1 = 0.0, d2 = 0.0;
  double4 wi = make_double4(0, 0, 0, 0);
  if (valid) {
    wi = w[i];
    const int64_t b1 = row[i + 1];
    int64_t b = row[i] + lane;
    auto bond = [&](const double4& gb, const double2& cb, const double4& wj) {
      const double w0 = wj.x - wi.x, w1 = wj.y - wi.y, w2 = wj.z - wi.z;
      const double sy = (wi.w + wj.w) + cb.x * (gb.x * w0 + gb.y * w1 + gb.z * w2);
      d0 += sy * gb.x + cb.y * w0;
      d1 += sy * gb.y + cb.y * w1;
      d2 += sy * gb.z + cb.y * w2;
    };
    for (; b + (kQsBatch2 - 1) * TPO < b1; b += kQsBatch2 * TPO) {  // batched as in k_qs_dtheta_g
      double4 gb[kQsBatch2], wj[kQsBatch2];
      double2 cb[kQsBatch2];
#pragma unroll
      for (int k = 0; k < kQsBatch2; ++k) gb[k] = ld_bond(g + b + k * TPO), cb[k] = __ldcs(gc + b + k * TPO);
#pragma unroll
      for (int k = 0; k < kQsBatch2; ++k) wj[k] = ld_w(w + bond_id(gb[k]));
#pragma unroll
      for (int k = 0; k < kQsBatch2; ++k) bond(gb[k], cb[k], wj[k]);
    }
    for (; b < b1; b += TPO) {
      const double4 gb = ld_bond(g + b);
      bond(gb, __ldcs(gc + b), ld_w(w + bond_id(gb)));
    }
  }
  d0 = qs_group_sum<TPO>(d0);
  d1 = qs_group_sum<TPO>(d1);
  d2 = qs_group_sum<TPO>(d2);
  double pq = 0.0;
  if (valid && lane < 3) {
    const double d = lane == 0 ? d0 : (lane == 1 ? d1 : d2);
    const double p = lane == 0 ? wi.x : (lane == 1 ? wi.y : wi.z);
    double kd = -xv[i].w * d;
    if (jm != 0.0) kd = jm * pt[i].w * p + jk * kd;  // implicit dynamics: (rho I + beta dt^2 K) p
    const double out = ((fixed[i] >> lane) & 1) ? p : kd;
    q[3 * i + lane] = out;
    pq = p * out;
  }
  double sum[1] = {pq};
  if (cg_grid_sum<1, kQsBlock>(sum, partial, &ctl->ticket[0]) && threadIdx.x == 0) ctl->pq = sum[0];
}

// Inverse 3x3 diagonal blocks of K (prescribed rows/columns set to identity).
__global__ void __launch_bounds__(kQsBlock) k_qs_block_diag(int64_t n, const int64_t* __restrict__ row,
                                                            const int32_t* __restrict__ col,
                                                            const uint8_t* __restrict__ dmg,
                                                            const double4* __restrict__ xv,
                                                            const double4* __restrict__ y,
                                                            const double4* __restrict__ ab,
                                                            const double4* __restrict__ pt,
                                                            const double* __restrict__ hp, int influence,
                                                            const uint8_t* __restrict__ fixed,
                                                            double* __restrict__ dinv, int invert, double jk = 1.0,
                                                            double jm = 0.0) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kQsTpo;
  const int lane = threadIdx.x & (kQsTpo - 1);
  const bool valid = i < n;
  double D[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  double hv[3] = {0, 0, 0};
  double4 xi = make_double4(0, 0, 0, 1), ai = make_double4(0, 0, 0, 0);
  double mi = 1.0;
  if (valid) {
    xi = xv[i];
    const double4 yi = y[i];
    ai = ab[i];
    mi = pt[i].x;
    const double h = hp[i];
    for (int64_t b = row[i] + lane; b < row[i + 1]; b += kQsTpo) {
      if (dmg[b]) continue;
      const int32_t j = col[b];
      const double4 xj = xv[j], yj = y[j], aj = ab[j];
      const double X0 = xj.x - xi.x, X1 = xj.y - xi.y, X2 = xj.z - xi.z;
      const double Y0 = yj.x - yi.x, Y1 = yj.y - yi.y, Y2 = yj.z - yi.z;
      const double zeta = sqrt(X0 * X0 + X1 * X1 + X2 * X2);
      const double dY = sqrt(Y0 * Y0 + Y1 * Y1 + Y2 * Y2);
      const double e = dY - zeta;
      const double om = qs_omega(influence, zeta, h);
      const double T = om * (zeta * (ai.x * ai.y + aj.x * aj.y) + (ai.z + aj.z) * e);
      const double V = xj.w;
      const double yh[3] = {Y0 / dY, Y1 / dY, Y2 / dY};
      const double a = -V * om * ((ai.z + aj.z) + 3.0 * om * zeta * zeta * aj.w * xi.w);
      const double g = -V * T / dY;
      for (int r = 0; r < 3; ++r) {
        hv[r] += V * om * zeta * yh[r];
        for (int c = 0; c < 3; ++c) D[3 * r + c] += (a - g) * yh[r] * yh[c] + (r == c ? g : 0.0);
      }
    }
  }
  for (int k = 0; k < 9; ++k) D[k] = qs_group_sum(D[k]);
  for (int k = 0; k < 3; ++k) hv[k] = qs_group_sum(hv[k]);
  if (valid && lane == 0) {
    const double s = 3.0 * ai.y / mi;
    double A[9];
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c) A[3 * r + c] = -xi.w * (D[3 * r + c] - s * hv[r] * hv[c]);  // K_ii = -V_i D_i
    if (jm != 0.0)  // implicit dynamics: blocks of rho I + beta dt^2 K
      for (int k = 0; k < 9; ++k) A[k] = jk * A[k] + ((k % 4 == 0) ? jm * pt[i].w : 0.0);
    const uint8_t fx = fixed[i];
    for (int c = 0; c < 3; ++c)
      if ((fx >> c) & 1)
        for (int k = 0; k < 3; ++k) {
          A[3 * c + k] = (k == c) ? 1.0 : 0.0;
          A[3 * k + c] = (k == c) ? 1.0 : 0.0;
        }
    if (!invert) {
      for (int k = 0; k < 9; ++k) dinv[9 * i + k] = A[k];
      return;
    }
    const double c00 = A[4] * A[8] - A[5] * A[7], c01 = A[5] * A[6] - A[3] * A[8], c02 = A[3] * A[7] - A[4] * A[6];
    const double det = A[0] * c00 + A[1] * c01 + A[2] * c02;
    const double id = 1.0 / det;
    double* o = dinv + 9 * i;
    o[0] = c00 * id;
    o[1] = (A[2] * A[7] - A[1] * A[8]) * id;
    o[2] = (A[1] * A[5] - A[2] * A[4]) * id;
    o[3] = c01 * id;
    o[4] = (A[0] * A[8] - A[2] * A[6]) * id;
    o[5] = (A[2] * A[3] - A[0] * A[5]) * id;
    o[6] = c02 * id;
    o[7] = (A[1] * A[6] - A[0] * A[7]) * id;
    o[8] = (A[0] * A[4] - A[1] * A[3]) * id;
  }
}

// z = P r (block Jacobi)
__global__ void k_qs_precond(int64_t n, const double* __restrict__ dinv, const double* __restrict__ r,
                             double* __restrict__ z) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double r0 = r[3 * i], r1 = r[3 * i + 1], r2 = r[3 * i + 2];
  const double* d = dinv + 9 * i;
  z[3 * i] = d[0] * r0 + d[1] * r1 + d[2] * r2;
  z[3 * i + 1] = d[3] * r0 + d[4] * r1 + d[5] * r2;
  z[3 * i + 2] = d[6] * r0 + d[7] * r1 + d[8] * r2;
}

// Partial dot products: out[3b] = a.b, out[3b+1] = a.c, out[3b+2] = a.a (c may equal b)
__global__ void k_qs_dots(int64_t m, const double* __restrict__ a, const double* __restrict__ b,
                          const double* __restrict__ c, double* __restrict__ partial) {
  __shared__ double s[3][kQsBlock];
  double ab = 0.0, ac = 0.0, aa = 0.0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
    const double va = a[k];
    ab += va * b[k];
    ac += va * c[k];
    aa += va * va;
  }
  s[0][threadIdx.x] = ab;
  s[1][threadIdx.x] = ac;
  s[2][threadIdx.x] = aa;
  __syncthreads();
  for (int o = kQsBlock / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o)
      for (int k = 0; k < 3; ++k) s[k][threadIdx.x] += s[k][threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 3; ++k) partial[3 * blockIdx.x + k] = s[k][0];
}

// x += alpha p ; r -= alpha q   (alpha = scal[0]/scal[1])
__global__ void k_qs_axpy2(int64_t m, const double* __restrict__ scal, const double4* __restrict__ w,
                           const double* __restrict__ q, double* __restrict__ x, double* __restrict__ r) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const double alpha = scal[0] / scal[1];
  const double4 p = w[k / 3];
  const int c = (int)(k % 3);
  const double pk = c == 0 ? p.x : (c == 1 ? p.y : p.z);
  x[k] += alpha * pk;
  r[k] -= alpha * q[k];
}

// p = z + beta p  with beta = scal[2]/scal[0] (flexible: (z.r - z.r_old)/rz_old folded by the host)
__global__ void k_qs_update_p(int64_t n, const double* __restrict__ scal, const double* __restrict__ z,
                              double4* __restrict__ w, int first) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4 p = w[i];
  if (first) {  // p = z; the previous direction is not read (it may be unset)
    p.x = z[3 * i];
    p.y = z[3 * i + 1];
    p.z = z[3 * i + 2];
  } else {
    const double beta = scal[3];
    p.x = z[3 * i] + beta * p.x;
    p.y = z[3 * i + 1] + beta * p.y;
    p.z = z[3 * i + 2] + beta * p.z;
  }
  w[i] = p;
}

// The learned preconditioner's scalars. scal: [0] r.z, [1] p.q, [3] beta,
// [4] r.r; red: [0] z.r, [2] r.r of the new residual, [4] z.q. what 0:
// scal[1] = p.q; else beta = max(0, z_new.(r_new - r_old)/rz_old) with
// z_new.r_old = z_new.r_new + alpha z_new.q (Polak-Ribiere).
__global__ void k_qs_set_scalars(double* scal, const double* red, int what) {
  if (threadIdx.x != 0) return;
  if (what == 0) {
    scal[1] = red[0];
  } else {
    const double rz_old = scal[0];
    const double alpha = __ddiv_rn(rz_old, scal[1]);
    const double zr_new = red[0];
    const double zr_old = __dadd_rn(zr_new, __dmul_rn(alpha, red[4]));
    const double beta = __ddiv_rn(__dsub_rn(zr_new, zr_old), rz_old);
    scal[3] = beta > 0.0 ? beta : 0.0;  // also 0 for a NaN beta
    scal[0] = zr_new;
    scal[2] = 0.0;
    scal[4] = red[2];
  }
}

__global__ void k_qs_axpy(int64_t m, double a, const double* __restrict__ x, double* __restrict__ y) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m) y[k] += a * x[k];
}

__global__ void k_qs_apply_bc(int64_t n, const uint8_t* __restrict__ mask, const double* __restrict__ a,
                              const double* __restrict__ b, const double2* __restrict__ fcp, double tc, double tp,
                              const double* __restrict__ u, double* __restrict__ du) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int c = 0; c < 3; ++c)
    if ((mask[i] >> c) & 1) {
      const int64_t k = 3 * i + c;
      // DirichletIncrementBC coeff 1 (Peridigm_BoundaryCondition.cpp:235); a
      // zero increment takes the previous value from the displacement
      // (:137-142); function dofs (mask bit 3 + c) from their values at the
      // two times (fcp)
      double cur, prev;
      if (fcp && ((mask[i] >> (c + 3)) & 1)) {
        cur = fcp[k].x, prev = fcp[k].y;
      } else {
        cur = a[k] * tc + b[k], prev = a[k] * tp + b[k];
      }
      const double d = cur - prev;
      du[k] = d == 0.0 ? cur - u[k] : d;
    }
}

__global__ void k_qs_finish(int64_t m, double inv_dt, const double* __restrict__ du, double* __restrict__ u,
                            double* __restrict__ v) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  u[k] += du[k];
  v[k] = du[k] * inv_dt;
}

// One CG iteration after the tangent passes, without a coarse level:
//   x += alpha p, r -= alpha q, z = P r (block Jacobi, or P = I), r.z, r.r
// with alpha = r.z / p.q, and the iteration's scalars from the last block.
// FIRST: the start of a solve (x and r as they are). One launch where the
// update, the preconditioner, the dot products, their reduction and the
// scalars were one each, with a copy of |r|^2 to the host.
template <bool FIRST>
__global__ void __launch_bounds__(kQsBlock) k_cg_update(int64_t n, const double4* __restrict__ w,
                                                        const double* __restrict__ q, double* __restrict__ x,
                                                        double* __restrict__ r, double* __restrict__ z,
                                                        const double* __restrict__ dinv, int use_bj,
                                                        double* __restrict__ partial, CgCtl* __restrict__ ctl) {
  if (!FIRST && ctl->state) return;
  const double alpha = FIRST ? 0.0 : ctl->rz / ctl->pq;
  double s[2] = {0.0, 0.0};
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double rv[3] = {r[3 * i], r[3 * i + 1], r[3 * i + 2]};
    if (!FIRST) {
      const double4 p = w[i];
      const double pv[3] = {p.x, p.y, p.z};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        rv[c] -= alpha * q[3 * i + c];
        r[3 * i + c] = rv[c];
        x[3 * i + c] += alpha * pv[c];
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double zc = rv[c];
      if (use_bj) {
        const double* d = dinv + 9 * i + 3 * c;
        zc = d[0] * rv[0] + d[1] * rv[1] + d[2] * rv[2];
      }
      z[3 * i + c] = zc;
      s[0] += rv[c] * zc;
      s[1] += rv[c] * rv[c];
    }
  }
  if (cg_grid_sum<2, kQsBlock>(s, partial, &ctl->ticket[1]) && threadIdx.x == 0) cg_scalars(ctl, s[0], s[1], FIRST);
}

// p = z + beta p (p = z at the start, where the previous direction may be unset)
__global__ void k_cg_direction(int64_t n, const double* __restrict__ z, double4* __restrict__ w, int first,
                               const CgCtl* __restrict__ ctl) {
  if (ctl->state) return;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double beta = ctl->beta;
  const double z0 = z[3 * i], z1 = z[3 * i + 1], z2 = z[3 * i + 2];
  if (first) {
    w[i] = make_double4(z0, z1, z2, 0.0);
  } else {
    const double4 p = w[i];
    w[i] = make_double4(z0 + beta * p.x, z1 + beta * p.y, z2 + beta * p.z, p.w);
  }
}

// ---------------------------------------------------------------------------
// A whole CG solve of a small body in one cooperative launch (no
// preconditioner or block Jacobi). Where every lane of the tangent passes is
// resident at once, an iteration is four phases between grid barriers: p
// published, q dtheta, K p with p.q, the update with the dot products. At some
// thousand points a phase is one or two round trips to L2, and the launches of
// the general loop cost as much again: 37x11x11 points, 63 us an iteration in
// eleven launches, 35 us in four, 21 us here. Lanes 0-2 of a point keep x, r and
// p of their component in registers; every block adds the blocks' partial sums
// in the same order, so all of them see the same scalars and stop together.
// ---------------------------------------------------------------------------
// A point's (p, q dtheta) that another block may have written before the last barrier.
__device__ __forceinline__ double4 ld_w_sync(const double4* p) {
  double4 r;
  asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];" : "=d"(r.x), "=d"(r.y), "=d"(r.z), "=d"(r.w) : "l"(p) : "memory");
  return r;
}

__device__ __forceinline__ double ld_t_sync(const double* p) {
  double r;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(p) : "memory");
  return r;
}

// Sums over the grid: this block's to partial[NV blk ..], a barrier, then all
// partials in block order. False when the barrier's wait ran out.
// Every warp adds the blocks' partials for itself (lane l those of blocks l,
// l + 32, ..), which saves a block barrier.
template <int NV>
__device__ __forceinline__ bool cg_sum_sync(double (&v)[NV], double* partial, unsigned int* bar, unsigned int& target,
                                            int* status) {
  __shared__ double sh[NV][32];
#pragma unroll
  for (int k = 0; k < NV; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if ((threadIdx.x & 31) == 0) sh[k][threadIdx.x >> 5] = v[k];
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double s = sh[threadIdx.x][0];
    for (unsigned w = 1; w < blockDim.x / 32; ++w) s += sh[threadIdx.x][w];
    partial[(size_t)NV * blockIdx.x + threadIdx.x] = s;
  }
  if (!grid_sync(bar, target, status)) return false;
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
#pragma unroll 5
  for (unsigned b = threadIdx.x & 31; b < gridDim.x; b += 32)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += __ldcg(partial + (size_t)NV * b + k);
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  return true;
}

struct CgSmallArgs {
  int64_t n;
  const int64_t* row;
  int slots;  // bonds per lane
  const double4* g;
  const double2* gc;
  const double4* ab;
  const double4* pt;
  const double4* xv;
  const uint8_t* fixed;
  const double* dinv;  // null: no preconditioner
  const double* r;     // right-hand side
  double* x;           // solution
  double4* w;
  double* t;           // q dtheta per point
  double* partial;
  double jk, jm, tol;
  long long max_it;
  CgCtl* ctl;
  unsigned int* bar;
  int* status;
};

// 16 lanes per point, one block per SM, the geometry of the lanes' bonds (G,
// k2, cx and the neighbor id) in shared memory.
constexpr int kCgLanes = 16, kCgSmallBlock = 512, kCgBond = 44;
__global__ void __launch_bounds__(kCgSmallBlock, 1) k_cg_small(CgSmallArgs A) {
  constexpr int L = kCgLanes, K = 4;
  extern __shared__ __align__(16) unsigned char cg_sm[];
  const int T = blockDim.x, tid = threadIdx.x, S = A.slots;
  double* sg = reinterpret_cast<double*>(cg_sm) + tid;  // bond t: G at sg[(3 t + c) T], k2 and cx at sk[2 t T], ..
  double* sk = sg + (size_t)3 * S * T;
  int32_t* sj = reinterpret_cast<int32_t*>(cg_sm + (size_t)40 * S * T) + tid;
  const int64_t i = ((int64_t)blockIdx.x * T + tid) / L;
  const int lane = tid & (L - 1);
  const bool valid = i < A.n, dof = valid && lane < 3;
  const int64_t ic = min(i, A.n - 1);
  double D[3] = {0.0, 0.0, 0.0};
  bool held = false;
  double r = 0.0, x = 0.0, p = 0.0;
  const double4 m = A.pt[ic];
  const double V = A.xv[ic].w, rho = m.w;
  double s = 0.0;  // (a point without bonds has q/m = 0/0, which its empty slots must not see)
  {
    const int64_t b0 = A.row[ic], b1 = A.row[ic + 1];
    if (b1 > b0) s = 3.0 * (A.ab[ic].y / m.x);
    for (int t = 0; t < S; ++t) {
      const int64_t b = b0 + lane + t * L;
      const bool in = valid && b < b1;
      const double4 gb = in ? ld_bond(A.g + b) : make_double4(0.0, 0.0, 0.0, __longlong_as_double(ic));
      const double2 kc = in ? A.gc[b] : make_double2(0.0, 0.0);
      sg[3 * t * T] = gb.x, sg[(3 * t + 1) * T] = gb.y, sg[(3 * t + 2) * T] = gb.z;
      sk[2 * t * T] = kc.x, sk[(2 * t + 1) * T] = kc.y;
      sj[t * T] = (int32_t)bond_id(gb);
    }
  }
  if (dof) {
    held = (A.fixed[i] >> lane) & 1;
    r = A.r[3 * i + lane];
#pragma unroll
    for (int c = 0; c < 3; ++c) D[c] = A.dinv ? A.dinv[9 * i + 3 * lane + c] : 0.0;
  }
  unsigned int target = 0;
  double* part_pq = A.partial + 2 * (size_t)gridDim.x;
  auto precond = [&](double rv) {  // lanes 0-2: their component of P r
    const double r0 = __shfl_sync(0xffffffffu, rv, 0, L), r1 = __shfl_sync(0xffffffffu, rv, 1, L),
                 r2 = __shfl_sync(0xffffffffu, rv, 2, L);
    return A.dinv ? D[0] * r0 + D[1] * r1 + D[2] * r2 : rv;
  };
  double z = precond(r);
  double dots[2] = {dof ? r * z : 0.0, dof ? r * r : 0.0};
  if (!cg_sum_sync<2>(dots, A.partial, A.bar, target, A.status)) return;
  const double rr0 = dots[1], r0 = sqrt(rr0);
  double rz = dots[0], rel = rr0 == 0.0 ? 0.0 : 1.0;
  int state = rr0 == 0.0 ? CG_ZERO_RHS : CG_RUNNING;
  long long it = 0;
  p = z;
  while (state == CG_RUNNING && it < A.max_it) {
    if (dof) (lane == 0 ? A.w[i].x : (lane == 1 ? A.w[i].y : A.w[i].z)) = p;
    const double p0 = __shfl_sync(0xffffffffu, p, 0, L), p1 = __shfl_sync(0xffffffffu, p, 1, L),
                 p2 = __shfl_sync(0xffffffffu, p, 2, L);
    if (!grid_sync(A.bar, target, A.status)) return;
    // tangent pass 1 (k_qs_dtheta_g), with the terms of pass 2 that p alone gives
    double acc = 0.0, d[3] = {0.0, 0.0, 0.0};
    for (int t0 = 0; t0 < S; t0 += K) {
      double4 wj[K];
#pragma unroll
      for (int k = 0; k < K; ++k) wj[k] = ld_w_sync(A.w + sj[(t0 + k < S ? t0 + k : t0) * T]);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (t0 + k < S) {
          const int t = t0 + k;
          const double G0 = sg[3 * t * T], G1 = sg[(3 * t + 1) * T], G2 = sg[(3 * t + 2) * T];
          const double w0 = wj[k].x - p0, w1 = wj[k].y - p1, w2 = wj[k].z - p2, cx = sk[(2 * t + 1) * T];
          const double gd = G0 * w0 + G1 * w1 + G2 * w2, kg = sk[2 * t * T] * gd;
          acc += gd;
          d[0] += kg * G0 + cx * w0;
          d[1] += kg * G1 + cx * w1;
          d[2] += kg * G2 + cx * w2;
        }
    }
    acc = s * qs_group_sum<L>(acc);
    if (valid && lane == 0) A.t[i] = acc;
    if (!grid_sync(A.bar, target, A.status)) return;
    // the rest of pass 2 (k_qs_df_g): (q dth_i + q dth_j) G
    for (int t0 = 0; t0 < S; t0 += 2 * K) {
      double tj[2 * K];
#pragma unroll
      for (int k = 0; k < 2 * K; ++k) tj[k] = ld_t_sync(A.t + sj[(t0 + k < S ? t0 + k : t0) * T]);
#pragma unroll
      for (int k = 0; k < 2 * K; ++k)
        if (t0 + k < S) {
          const int t = t0 + k;
          const double ts = acc + tj[k];
          d[0] += ts * sg[3 * t * T];
          d[1] += ts * sg[(3 * t + 1) * T];
          d[2] += ts * sg[(3 * t + 2) * T];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) d[c] = qs_group_sum<L>(d[c]);
    double q = 0.0;
    if (dof) {
      q = -V * (lane == 0 ? d[0] : (lane == 1 ? d[1] : d[2]));
      if (A.jm != 0.0) q = A.jm * rho * p + A.jk * q;  // implicit dynamics: (rho I + beta dt^2 K) p
      if (held) q = p;
    }
    double pq[1] = {dof ? p * q : 0.0};
    if (!cg_sum_sync<1>(pq, part_pq, A.bar, target, A.status)) return;
    const double alpha = rz / pq[0];
    x += alpha * p;
    r -= alpha * q;
    z = precond(r);
    dots[0] = dof ? r * z : 0.0;
    dots[1] = dof ? r * r : 0.0;
    if (!cg_sum_sync<2>(dots, A.partial, A.bar, target, A.status)) return;
    rel = sqrt(dots[1]) / r0;
    ++it;
    if (!isfinite(rel)) state = CG_NONFINITE;
    else if (rel <= A.tol) state = CG_CONVERGED;
    p = z + (dots[0] / rz) * p;
    rz = dots[0];
  }
  if (state == CG_RUNNING) state = CG_MAX_ITERATIONS;
  if (dof) A.x[3 * i + lane] = x;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.ctl->it = it;
    A.ctl->rel = rel;
    A.ctl->state = state;
  }
}

// The start of a solve (state, tolerance, where the report goes).
__global__ void k_cg_begin(CgCtl* ctl, double tol, long long max_it, CgReport* report) {
  ctl->state = CG_RUNNING;
  ctl->ticket[0] = ctl->ticket[1] = 0;
  ctl->tol = tol;
  ctl->max_it = max_it;
  ctl->it = 0;
  ctl->report = report;
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
static unsigned g1(int64_t m) { return (unsigned)((m + kQsBlock - 1) / kQsBlock); }
static unsigned gt(int64_t n, int tpo = kQsTpo) { return (unsigned)((n * tpo + kQsBlock - 1) / kQsBlock); }
// Blocks of the CG vector kernels: enough to fill the chip, few enough that
// the last block adds their sums quickly.
static unsigned gv(int64_t n) { return std::min(g1(n), 4u * 148u); }
// Lanes per point of the tangent passes.
static int qs_lanes(int64_t n) { return n <= kQsWide ? 32 : kQsTpo; }

static int qs_alloc(pd_ctx* c) {
  if (!c->qs) c->qs = new QsState();
  QsState* s = c->qs;
  if (s->n == c->n) return PD_OK;
  const int64_t n = c->n;
  PD_CUDA_TRY(c, s->yq.alloc(n));
  PD_CUDA_TRY(c, s->abq.alloc(n));
  PD_CUDA_TRY(c, s->w.alloc(n));
  PD_CUDA_TRY(c, s->th.alloc(n));
  PD_CUDA_TRY(c, s->nd.alloc(n));
  for (auto* b : {&s->f, &s->r, &s->du, &s->x, &s->z, &s->q, &s->pred}) PD_CUDA_TRY(c, b->alloc(3 * n));
  PD_CUDA_TRY(c, s->dinv.alloc(9 * n));
  PD_CUDA_TRY(c, s->partial.alloc(3 * (size_t)std::max<int64_t>(kRedBlocks, gt(n, qs_lanes(n))) + 8));
  PD_CUDA_TRY(c, s->ctl.alloc(1));
  PD_CUDA_TRY(c, dzero(c, s->ctl.p, s->ctl.bytes()));
  PD_CUDA_TRY(c, s->scal.alloc(16));
  PD_CUDA_TRY(c, s->fixed.alloc(n));
  PD_CUDA_TRY(c, dzero(c, s->pred.p, s->pred.bytes()));
  s->small_threads = -1;
  s->n = n;
  return PD_OK;
}

// Whether there is a word for solves to report through. A page registered with
// the driver: 0.4 ms for a context's first solve, where cudaHostAlloc took 1.9
// to 2.6 ms; the one-launch solve needs none. Where the page cannot be had, the
// host reads the solve's record after every iteration.
static bool qs_report(pd_ctx* c) {
  QsState* s = c->qs;
  if (s->report || s->no_report) return s->report != nullptr;
  constexpr size_t kPage = 4096;
  void* page = aligned_alloc(kPage, kPage);
  if (page && cudaHostRegister(page, kPage, cudaHostRegisterMapped) == cudaSuccess) {
    if (cudaHostGetDevicePointer((void**)&s->report_dev, page, 0) == cudaSuccess) {
      s->report = (CgReport*)page;
      return true;
    }
    cudaHostUnregister(page);
  }
  cudaGetLastError();
  free(page);
  s->report_dev = nullptr;
  s->no_report = true;
  return false;
}

const uint8_t* qs_fixed_mask(const pd_ctx* c) { return c->qs ? c->qs->fixed.p : nullptr; }

void qs_release(pd_ctx* c) {
  delete c->qs;
  c->qs = nullptr;
}

// Residual at y = x + u + du; returns ||r||_2 and ||r||_inf.
static int qs_residual(pd_ctx* c, double* l2, double* linf) {
  QsState* s = c->qs;
  const int64_t n = c->n;
  k_qs_positions<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->xv.p, c->u.p, s->du.p, s->yq.p);
  PD_CUDA_TRY(c, launch_fp64_eval_at(c, s->yq.p, s->abq.p, s->th.p, s->nd.p, s->f.p));
  s->geo_dirty = true;
  k_qs_residual<<<kRedBlocks, kQsBlock, 0, c->stream>>>(n, s->f.p, c->xv.p, s->fixed.p, s->r.p, s->partial.p);
  k_qs_reduce<<<1, kQsBlock, 0, c->stream>>>(s->partial.p, kRedBlocks, 2, 1, s->scal.p + 8);
  PD_CUDA_TRY(c, cudaGetLastError());
  double h[2];
  PD_CUDA_TRY(c, cudaMemcpyAsync(h, s->scal.p + 8, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  PD_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  *l2 = std::sqrt(h[0]);
  *linf = h[1];
  if (!std::isfinite(*l2)) {
    c->err = "NaN returned by force evaluation";
    return PD_ERR_NONFINITE;
  }
  return PD_OK;
}

// z = M r of the learned preconditioner: block Jacobi, the network's
// correction and, where it is on, the coarse one.
static int qs_apply_learned(pd_ctx* c, const double* r, double* z) {
  QsState* s = c->qs;
  k_qs_precond<<<g1(c->n), kQsBlock, 0, c->stream>>>(c->n, s->dinv.p, r, z);
  PD_CUDA_TRY(c, cudaGetLastError());
  TRY_RC(mpnn_apply_add(c, r, z));
  if (s->coarse_on) TRY_RC(coarse_apply_add(c, r, z, s->fixed.p));
  return PD_OK;
}

// Tangent-vector product q = K w.xyz (w.w receives q dtheta) on the per-bond
// geometry, rebuilt first when the state changed.
static int qs_geometry(pd_ctx* c) {
  QsState* s = c->qs;
  const int64_t n = c->n;
  if (s->geo_dirty || s->gco.count < (size_t)c->nb) {
    if (s->gco.count < (size_t)c->nb) {
      PD_CUDA_TRY(c, s->geo.alloc((size_t)c->nb));
      PD_CUDA_TRY(c, s->gco.alloc((size_t)c->nb));
    }
    k_qs_bond_geom<<<gt(n), kQsBlock, 0, c->stream>>>(n, c->row.p, c->col.p, c->dmg.p, c->xv.p, s->yq.p, s->abq.p,
                                                      c->hp.p, c->influence, s->geo.p, s->gco.p);
    s->geo_dirty = false;
  }
  PD_CUDA_TRY(c, cudaGetLastError());
  return PD_OK;
}

template <int TPO>
static void launch_tangent(pd_ctx* c) {
  QsState* s = c->qs;
  const int64_t n = c->n;
  k_qs_dtheta_g<TPO><<<gt(n, TPO), kQsBlock, 0, c->stream>>>(n, c->row.p, s->geo.p, s->abq.p, c->pt.p,
                                                             s->w.p, s->ctl.p);
  k_qs_df_g<TPO><<<gt(n, TPO), kQsBlock, 0, c->stream>>>(n, c->row.p, s->geo.p, s->gco.p, c->xv.p, s->w.p,
                                                         s->fixed.p, s->q.p, s->partial.p, c->pt.p, s->jk, s->jm,
                                                         s->ctl.p);
}

static int qs_tangent(pd_ctx* c) {
  TRY_RC(qs_geometry(c));
  if (qs_lanes(c->n) == 32) launch_tangent<32>(c);
  else launch_tangent<kQsTpo>(c);
  PD_CUDA_TRY(c, cudaGetLastError());
  return PD_OK;
}

// Outside a solve the passes must not see the last one's end.
static int qs_tangent_alone(pd_ctx* c) {
  QsState* s = c->qs;
  k_cg_begin<<<1, 1, 0, c->stream>>>(s->ctl.p, 0.0, 0, s->report_dev);
  return qs_tangent(c);
}

// Preconditioned CG on K x = r (Belos BlockCG in the reference). Flexible
// (Polak-Ribiere) beta when the preconditioner is not a fixed linear operator.
__global__ void k_qs_true_residual(int64_t m, const double* __restrict__ b, const double* __restrict__ q,
                                   double* __restrict__ r) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m) r[k] = b[k] - q[k];
}

__global__ void k_qs_x_to_w(int64_t n, const double* __restrict__ x, double4* __restrict__ w) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  w[i] = make_double4(x[3 * i], x[3 * i + 1], x[3 * i + 2], 0.0);
}

static void k_qs_pack_x(int64_t n, QsState* s, pd_ctx* c) {
  k_qs_x_to_w<<<g1(n), kQsBlock, 0, c->stream>>>(n, s->x.p, s->w.p);
}

static int qs_cg_run(pd_ctx* c, int precond, double rel_tol, int max_it, int* iters, double* rel_out);
static int qs_cg_flexible(pd_ctx* c, double rel_tol, int max_it, int* iters, double* rel_out, bool* stalled);
constexpr int kCgAhead = 3;  // iterations the host launches ahead of the last one reported

// CG with the learned preconditioner first and 3x3 block Jacobi (the
// reference's "Block 3x3") as the fallback: when the flexible iteration
// stalls, or when the true FP64 residual |b - K x| (recomputed, not the
// recursive one) misses the tolerance, the solve restarts from the current x
// with block Jacobi. The true residual decides.
static int qs_cg(pd_ctx* c, int precond, double rel_tol, int max_it, int* iters, double* rel_out) {
  QsState* s = c->qs;
  const int64_t m = 3 * c->n;
  if (precond != PD_PRECOND_MPNN) return qs_cg_run(c, precond, rel_tol, max_it, iters, rel_out);
  if (s->cg_b.count < (size_t)m) PD_CUDA_TRY(c, s->cg_b.alloc(m));
  if (s->cg_x0.count < (size_t)m) PD_CUDA_TRY(c, s->cg_x0.alloc(m));
  DBuf<double>& b = s->cg_b;
  DBuf<double>& x0 = s->cg_x0;
  PD_CUDA_TRY(c, cudaMemcpyAsync(b.p, s->r.p, m * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  bool stalled = false;
  int its = 0;
  double rel = 0.0;
  int rc = qs_cg_flexible(c, rel_tol, max_it, &its, &rel, &stalled);
  if (rc != PD_OK && rc != PD_ERR_NOT_CONVERGED && rc != PD_ERR_NONFINITE) return rc;
  TRY_RC(mpnn_check_status(c));
  // true residual r = b - K x
  const int64_t n = c->n;
  k_qs_pack_x(n, s, c);
  TRY_RC(qs_tangent_alone(c));
  k_qs_true_residual<<<g1(m), kQsBlock, 0, c->stream>>>(m, b.p, s->q.p, s->r.p);
  k_qs_dots<<<kRedBlocks, kQsBlock, 0, c->stream>>>(m, s->r.p, s->r.p, b.p, s->partial.p);
  k_qs_reduce<<<1, kQsBlock, 0, c->stream>>>(s->partial.p, kRedBlocks, 3, 0, s->scal.p + 8);
  double h[3];
  PD_CUDA_TRY(c, cudaMemcpyAsync(h, s->scal.p + 8, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  k_qs_dots<<<kRedBlocks, kQsBlock, 0, c->stream>>>(m, b.p, b.p, b.p, s->partial.p);
  k_qs_reduce<<<1, kQsBlock, 0, c->stream>>>(s->partial.p, kRedBlocks, 3, 0, s->scal.p + 12);
  double hb[3];
  PD_CUDA_TRY(c, cudaMemcpyAsync(hb, s->scal.p + 12, sizeof(hb), cudaMemcpyDeviceToHost, c->stream));
  PD_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  const double true_rel = hb[0] > 0 ? std::sqrt(h[0] / hb[0]) : 0.0;

  if (std::isfinite(true_rel) && true_rel <= rel_tol && !stalled) {
    *iters = its;
    *rel_out = true_rel;
    return PD_OK;
  }
  // fall back: block Jacobi on the remaining system K dx = b - K x (x kept when finite)
  c->qs_fallbacks += 1;
  if (!std::isfinite(true_rel)) {
    PD_CUDA_TRY(c, cudaMemsetAsync(s->x.p, 0, m * sizeof(double), c->stream));
    PD_CUDA_TRY(c, cudaMemcpyAsync(s->r.p, b.p, m * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  }
  PD_CUDA_TRY(c, cudaMemcpyAsync(x0.p, s->x.p, m * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  // the remaining system is solved to the tolerance relative to |b|
  const double tol2 = (std::isfinite(true_rel) && true_rel > 0) ? std::min(1.0, rel_tol / true_rel) : rel_tol;
  int its2 = 0;
  double rel2 = 0.0;
  rc = qs_cg_run(c, PD_PRECOND_BLOCK_JACOBI, tol2, max_it, &its2, &rel2);
  k_qs_axpy<<<g1(m), kQsBlock, 0, c->stream>>>(m, 1.0, x0.p, s->x.p);
  PD_CUDA_TRY(c, cudaGetLastError());
  *iters = its + its2;
  *rel_out = rel2 * (std::isfinite(true_rel) && true_rel > 0 ? true_rel : 1.0);
  return rc;
}

// CG with the learned preconditioner (flexible beta), one host read per iteration.
static int qs_cg_flexible(pd_ctx* c, double rel_tol, int max_it, int* iters, double* rel_out, bool* stalled) {
  QsState* s = c->qs;
  const int64_t n = c->n, m = 3 * n;
  double best = 1.0;
  int best_it = 0;
  *stalled = false;
  PD_CUDA_TRY(c, cudaMemsetAsync(s->x.p, 0, s->x.bytes(), c->stream));
  k_cg_begin<<<1, 1, 0, c->stream>>>(s->ctl.p, 0.0, 0, s->report_dev);
  TRY_RC(qs_apply_learned(c, s->r.p, s->z.p));
  // scal: [0] rz, [1] pq, [3] beta, [4] rr
  k_qs_dots<<<kRedBlocks, kQsBlock, 0, c->stream>>>(m, s->r.p, s->z.p, s->z.p, s->partial.p);
  k_qs_reduce<<<1, kQsBlock, 0, c->stream>>>(s->partial.p, kRedBlocks, 3, 0, s->scal.p + 8);
  double h[3];
  PD_CUDA_TRY(c, cudaMemcpyAsync(h, s->scal.p + 8, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  PD_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  const double r0 = std::sqrt(h[2]);
  const double rz = h[0];
  *iters = 0;
  *rel_out = 0.0;
  if (r0 == 0.0) return PD_OK;
  PD_CUDA_TRY(c, cudaMemcpyAsync(s->scal.p, &rz, sizeof(double), cudaMemcpyHostToDevice, c->stream));
  k_qs_update_p<<<g1(n), kQsBlock, 0, c->stream>>>(n, s->scal.p, s->z.p, s->w.p, 1);
  double rel = 1.0;
  int it = 0;
  while (it < max_it) {
    TRY_RC(qs_tangent(c));
    k_qs_set_scalars<<<1, 32, 0, c->stream>>>(s->scal.p, &s->ctl.p->pq, 0);
    k_qs_axpy2<<<g1(m), kQsBlock, 0, c->stream>>>(m, s->scal.p, s->w.p, s->q.p, s->x.p, s->r.p);
    TRY_RC(qs_apply_learned(c, s->r.p, s->z.p));
    k_qs_dots<<<kRedBlocks, kQsBlock, 0, c->stream>>>(m, s->r.p, s->z.p, s->z.p, s->partial.p);
    k_qs_reduce<<<1, kQsBlock, 0, c->stream>>>(s->partial.p, kRedBlocks, 3, 0, s->scal.p + 8);
    // z_new.q for beta = z_new.(r_new - r_old)/rz_old, r_old = r_new + alpha q
    k_qs_dots<<<kRedBlocks, kQsBlock, 0, c->stream>>>(m, s->z.p, s->q.p, s->q.p, s->partial.p);
    k_qs_reduce<<<1, kQsBlock, 0, c->stream>>>(s->partial.p, kRedBlocks, 3, 0, s->scal.p + 12);
    k_qs_set_scalars<<<1, 32, 0, c->stream>>>(s->scal.p, s->scal.p + 8, 1);
    double rr;  // the only host read of the iteration: |r|^2 for the stopping test
    PD_CUDA_TRY(c, cudaMemcpyAsync(&rr, s->scal.p + 4, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    PD_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
    rel = std::sqrt(rr) / r0;
    ++it;
    if (!std::isfinite(rel)) {
      c->err = "CG diverged (non-finite residual)";
      return PD_ERR_NONFINITE;
    }
    if (rel <= rel_tol) break;
    // stall: no 10x decrease of the residual over 60 iterations
    if (rel < 0.1 * best) best = rel, best_it = it;
    if (it - best_it > 60) {
      *stalled = true;
      break;
    }
    k_qs_update_p<<<g1(n), kQsBlock, 0, c->stream>>>(n, s->scal.p, s->z.p, s->w.p, 0);
  }
  PD_CUDA_TRY(c, cudaGetLastError());
  *iters = it;
  *rel_out = rel;
  return rel <= rel_tol ? PD_OK : PD_ERR_NOT_CONVERGED;
}

// Waits until the solve has reported `it` iterations or its end. The report
// is written by kernels already in the stream: the wait ends with them (or
// with their error, or when the stream is idle and nothing was reported).
static int cg_wait(pd_ctx* c, long long it, CgReport* out) {
  const volatile CgReport* h = c->qs->report;
  bool idle = false;
  for (unsigned spin = 0;; ++spin) {
    const CgReport word = *h;
    if (word != ~0ull && ((word & 7) != CG_RUNNING || (long long)(word >> 3) >= it)) {
      *out = word;
      return PD_OK;
    }
    if (idle) {
      c->err = "the CG solve stopped without a report";
      return PD_ERR_CUDA;
    }
    if ((spin & 1023u) == 1023u) {
      const cudaError_t e = cudaStreamQuery(c->stream);
      if (e == cudaSuccess) idle = true;  // one more look at the report
      else if (e != cudaErrorNotReady) PD_CUDA_TRY(c, e);
    }
  }
}

// The same from the solve's record, after what is in the stream.
static int cg_read(pd_ctx* c, CgReport* out) {
  CgCtl h{};
  PD_CUDA_TRY(c, d2h(c, &h, c->qs->ctl.p, sizeof(h)));
  *out = (CgReport)h.it * 8 + h.state;
  return PD_OK;
}

// Threads per block of the one-launch solve; 0 when the body's lanes are not
// all resident with their geometry in shared memory (about 4,500 points of 110
// bonds), or the device takes no cooperative launches.
static int cg_small_threads(pd_ctx* c) {
  QsState* s = c->qs;
  if (s->small_threads < 0 || s->small_max_row != c->max_row) {
    s->small_threads = 0;
    s->small_max_row = c->max_row;
    int sms = 0, coop = 0, smem = 0, per = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device) != cudaSuccess ||
        cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device) != cudaSuccess || !coop)
      return 0;
    const int64_t threads = ((c->n * kCgLanes + sms - 1) / sms + 31) / 32 * 32;
    const int64_t slots = std::max(1, (c->max_row + kCgLanes - 1) / kCgLanes), bytes = threads * slots * kCgBond;
    if (threads > kCgSmallBlock || bytes > smem - 2048) return 0;
    // (one value for every context, whatever it needs: the attribute is the kernel's)
    if (cudaFuncSetAttribute(k_cg_small, cudaFuncAttributeMaxDynamicSharedMemorySize, smem - 2048) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cg_small, (int)threads, (size_t)bytes) != cudaSuccess ||
        per < 1) {
      cudaGetLastError();
      return 0;
    }
    s->small_threads = (int)threads;
    s->small_slots = (int)slots;
    c->cg_bytes = (int)bytes;
  }
  return s->small_threads;
}

// *taken: false when the driver refuses the launch; nothing has run then.
static int cg_run_small(pd_ctx* c, int precond, double rel_tol, int max_it, int* iters, double* rel_out, int threads,
                        bool* taken) {
  QsState* s = c->qs;
  TRY_RC(qs_geometry(c));
  if (c->small_bar.count < 1) PD_CUDA_TRY(c, c->small_bar.alloc(1));
  PD_CUDA_TRY(c, cudaMemsetAsync(c->small_bar.p, c->bar_fill, sizeof(unsigned int), c->stream));
  PD_CUDA_TRY(c, dzero(c, s->ctl.p, s->ctl.bytes()));
  CgSmallArgs A{};
  A.n = c->n;
  A.row = c->row.p;
  A.slots = s->small_slots;
  A.g = s->geo.p;
  A.gc = s->gco.p;
  A.ab = s->abq.p;
  A.pt = c->pt.p;
  A.xv = c->xv.p;
  A.fixed = s->fixed.p;
  A.dinv = precond == PD_PRECOND_NONE ? nullptr : s->dinv.p;
  A.r = s->r.p;
  A.x = s->x.p;
  A.w = s->w.p;
  A.t = s->z.p;
  A.partial = s->partial.p;
  A.jk = s->jk;
  A.jm = s->jm;
  A.tol = rel_tol;
  A.max_it = max_it;
  A.ctl = s->ctl.p;
  A.bar = c->small_bar.p;
  A.status = &s->ctl.p->waits;
  void* args[] = {&A};
  *taken = cudaLaunchCooperativeKernel((const void*)&k_cg_small,
                                       dim3((unsigned)((c->n * kCgLanes + threads - 1) / threads)), dim3(threads), args,
                                       (size_t)c->cg_bytes, c->stream) == cudaSuccess;
  if (!*taken) {
    cudaGetLastError();  // (an earlier fault comes up again at the next call)
    s->small_threads = 0;
    return PD_OK;
  }
  CgCtl h{};
  PD_CUDA_TRY(c, d2h(c, &h, s->ctl.p, sizeof(h)));
  *iters = (int)h.it;
  *rel_out = h.rel;
  if (h.waits & ST_TIMEOUT) {  // (whatever the others found: not every point has its x)
    c->err = "a bounded device wait ran out in the CG solve";
    return PD_ERR_TIMEOUT;
  }
  switch (h.state) {
    case CG_CONVERGED:
    case CG_ZERO_RHS: return PD_OK;
    case CG_NONFINITE: c->err = "CG diverged (non-finite residual)"; return PD_ERR_NONFINITE;
    default: return PD_ERR_NOT_CONVERGED;
  }
}

// CG with a fixed preconditioner (none, block Jacobi, two-level): the scalars
// and the stopping test stay on the device, and the host runs kCgAhead
// iterations ahead of the last one reported. Launches after the end of the
// solve return at once.
static int qs_cg_run(pd_ctx* c, int precond, double rel_tol, int max_it, int* iters, double* rel_out) {
  QsState* s = c->qs;
  const int64_t n = c->n;
  const int every = mpnn_capture_every(c) && precond != PD_PRECOND_NONE ? mpnn_capture_every(c) : 0;
  const bool coarse = s->coarse_on && precond == PD_PRECOND_TWO_LEVEL;
  const int use_bj = precond != PD_PRECOND_NONE;
  if (!coarse && every == 0) {
    const int threads = cg_small_threads(c);
    bool taken = false;
    if (threads) TRY_RC(cg_run_small(c, precond, rel_tol, max_it, iters, rel_out, threads, &taken));
    if (taken) return PD_OK;
  }
  const bool follow = qs_report(c);
  const int ahead = every > 0 || !follow ? 0 : kCgAhead;  // training pairs are taken at the reported iterate
  auto update = [&](bool first) -> int {
    if (coarse)
      return coarse_cg_update(c, s->w.p, s->q.p, s->x.p, s->r.p, s->z.p, s->dinv.p, s->fixed.p, s->partial.p, s->ctl.p,
                              first, gv(n));
    if (first)
      k_cg_update<true><<<gv(n), kQsBlock, 0, c->stream>>>(n, s->w.p, s->q.p, s->x.p, s->r.p, s->z.p, s->dinv.p,
                                                           use_bj, s->partial.p, s->ctl.p);
    else
      k_cg_update<false><<<gv(n), kQsBlock, 0, c->stream>>>(n, s->w.p, s->q.p, s->x.p, s->r.p, s->z.p, s->dinv.p,
                                                            use_bj, s->partial.p, s->ctl.p);
    return PD_OK;
  };
  if (follow) *(volatile CgReport*)s->report = ~0ull;  // (no kernel of an earlier solve is in flight: each ends with a wait for the stream)
  PD_CUDA_TRY(c, cudaMemsetAsync(s->x.p, 0, s->x.bytes(), c->stream));
  k_cg_begin<<<1, 1, 0, c->stream>>>(s->ctl.p, rel_tol, max_it, s->report_dev);
  TRY_RC(update(true));
  k_cg_direction<<<g1(n), kQsBlock, 0, c->stream>>>(n, s->z.p, s->w.p, 1, s->ctl.p);
  if (every > 0) TRY_RC(mpnn_snapshot(c, s->r.p, s->x.p));
  CgReport at = 0;
  int rc = PD_OK;
  for (int it = 1; it <= max_it; ++it) {
    rc = qs_tangent(c);
    if (rc == PD_OK) rc = update(false);
    PD_CUDA_TRY(c, cudaGetLastError());
    if (rc == PD_OK) rc = follow ? cg_wait(c, it - ahead, &at) : cg_read(c, &at);
    if (rc != PD_OK || (at & 7) != CG_RUNNING) break;
    if (every > 0 && it % every == 0) TRY_RC(mpnn_snapshot(c, s->r.p, s->x.p));
    k_cg_direction<<<g1(n), kQsBlock, 0, c->stream>>>(n, s->z.p, s->w.p, 0, s->ctl.p);
  }
  if (rc == PD_OK && follow && (at & 7) == CG_RUNNING) rc = cg_wait(c, max_it, &at);
  // (the copy also ends the launches beyond the last iteration, which must not
  // reach into the next solve's report)
  const cudaError_t e = d2h(c, rel_out, &s->ctl.p->rel, sizeof(double));
  if (rc != PD_OK) {
    if (every > 0) mpnn_drop_snapshots(c);
    return rc;
  }
  PD_CUDA_TRY(c, e);
  const int state = (int)(at & 7);
  *iters = (int)(at >> 3);
  if (state == CG_NONFINITE) {
    if (every > 0) mpnn_drop_snapshots(c);
    c->err = "CG diverged (non-finite residual)";
    return PD_ERR_NONFINITE;
  }
  if (state == CG_ZERO_RHS) {
    if (every > 0) mpnn_drop_snapshots(c);
    return PD_OK;
  }
  if (every > 0) {
    if (state == CG_CONVERGED) TRY_RC(mpnn_commit_snapshots(c, s->x.p, s->dinv.p));
    else mpnn_drop_snapshots(c);
  }
  return state == CG_CONVERGED ? PD_OK : PD_ERR_NOT_CONVERGED;
}

__global__ void k_qs_pack_w(int64_t n, const double* __restrict__ w, const uint8_t* __restrict__ fixed,
                            double4* __restrict__ w4) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint8_t f = fixed[i];
  w4[i] = make_double4((f & 1) ? 0.0 : w[3 * i], (f & 2) ? 0.0 : w[3 * i + 1], (f & 4) ? 0.0 : w[3 * i + 2], 0.0);
}

__global__ void k_qs_fixed_rows(int64_t n, const double* __restrict__ w, const uint8_t* __restrict__ fixed,
                                double* __restrict__ q) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int c = 0; c < 3; ++c)
    if ((fixed[i] >> c) & 1) q[3 * i + c] = w[3 * i + c];
}

static int qs_prepare_at(pd_ctx* c, const double* u_dev) {
  TRY_RC(ensure_ready_internal(c));
  if (c->material_model != PD_MATERIAL_LPS) {
    c->err = "the quasi-static solve supports the LPS material model only";
    return PD_ERR_UNSUPPORTED;
  }
  if (c->phantoms) {
    c->err = "the implicit and quasi-static solves need symmetric bond families (one horizon across the blocks)";
    return PD_ERR_UNSUPPORTED;
  }
  TRY_RC(qs_alloc(c));
  QsState* s = c->qs;
  const int64_t n = c->n;
  std::vector<uint8_t> fx(n, 0);
  for (int64_t i = 0; i < n; ++i) fx[i] = c->h_bc_mask.empty() ? 0 : (uint8_t)(c->h_bc_mask[i] & 7);  // the coordinates held
  PD_CUDA_TRY(c, cudaMemcpyAsync(s->fixed.p, fx.data(), n, cudaMemcpyHostToDevice, c->stream));
  PD_CUDA_TRY(c, cudaMemsetAsync(s->du.p, 0, 3 * n * sizeof(double), c->stream));
  k_qs_positions<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->xv.p, u_dev, s->du.p, s->yq.p);
  PD_CUDA_TRY(c, launch_fp64_eval_at(c, s->yq.p, s->abq.p, s->th.p, s->nd.p, s->f.p));
  s->geo_dirty = true;
  k_qs_qm<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->pt.p, s->abq.p);
  PD_CUDA_TRY(c, cudaGetLastError());
  return PD_OK;
}

// Matrix-free tangent K w at displacement u (prescribed rows/columns identity).
int qs_tangent_apply(pd_ctx* c, const double* u_dev, const double* w_dev, double* kw_dev) {
  TRY_RC(qs_prepare_at(c, u_dev));
  QsState* s = c->qs;
  const int64_t n = c->n;
  k_qs_pack_w<<<g1(n), kQsBlock, 0, c->stream>>>(n, w_dev, s->fixed.p, s->w.p);
  TRY_RC(qs_tangent_alone(c));
  k_qs_fixed_rows<<<g1(n), kQsBlock, 0, c->stream>>>(n, w_dev, s->fixed.p, s->q.p);
  PD_CUDA_TRY(c, cudaMemcpyAsync(kw_dev, s->q.p, 3 * n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  return PD_OK;
}

// 3x3 diagonal blocks of K at displacement u (row-major, 9 per point).
int qs_tangent_blocks(pd_ctx* c, const double* u_dev, double* blocks_dev) {
  TRY_RC(qs_prepare_at(c, u_dev));
  QsState* s = c->qs;
  const int64_t n = c->n;
  k_qs_block_diag<<<gt(n), kQsBlock, 0, c->stream>>>(n, c->row.p, c->col.p, c->dmg.p, c->xv.p, s->yq.p, s->abq.p,
                                                     c->pt.p, c->hp.p, c->influence, s->fixed.p, blocks_dev, 0);
  PD_CUDA_TRY(c, cudaGetLastError());
  return PD_OK;
}

// Tangent at the context's current displacement, for repeated products.
int qs_prepare_current(pd_ctx* c) { return qs_prepare_at(c, c->u.p); }

// Block-Jacobi inverse blocks at the tangent prepared by qs_prepare_current.
int qs_block_jacobi_current(pd_ctx* c, const double** dinv_out) {
  QsState* s = c->qs;
  const int64_t n = c->n;
  k_qs_block_diag<<<gt(n), kQsBlock, 0, c->stream>>>(n, c->row.p, c->col.p, c->dmg.p, c->xv.p, s->yq.p, s->abq.p,
                                                     c->pt.p, c->hp.p, c->influence, s->fixed.p, s->dinv.p, 1);
  PD_CUDA_TRY(c, cudaGetLastError());
  *dinv_out = s->dinv.p;
  return PD_OK;
}

// Coarse operator at the tangent prepared by qs_prepare_current.
int qs_build_coarse_current(pd_ctx* c, double cell) {
  QsState* s = c->qs;
  TRY_RC(coarse_build(c, s->yq.p, s->abq.p, s->fixed.p, cell, nullptr));
  s->coarse_on = true;
  s->coarse_rebuild = true;  // the next load step builds its own
  return PD_OK;
}

// Coarse space at displacement u: size, aggregates, assembled matrix and inverse (device buffers, may be null).
int qs_coarse_operator(pd_ctx* c, const double* u_dev, double cell, int64_t* n_coarse, int32_t* agg_dev,
                       double* A_dev, double* Ainv_dev) {
  TRY_RC(qs_prepare_at(c, u_dev));
  QsState* s = c->qs;
  TRY_RC(coarse_build(c, s->yq.p, s->abq.p, s->fixed.p, cell, A_dev));
  s->coarse_rebuild = true;
  *n_coarse = coarse_size(c);
  if (agg_dev) TRY_RC(coarse_aggregates(c, agg_dev));
  if (Ainv_dev) TRY_RC(coarse_copy_inverse(c, Ainv_dev));
  PD_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  return PD_OK;
}

// kw = K w with the tangent prepared by qs_prepare_current.
int qs_apply_K(pd_ctx* c, const double* w_dev, double* kw_dev) {
  QsState* s = c->qs;
  const int64_t n = c->n;
  k_qs_pack_w<<<g1(n), kQsBlock, 0, c->stream>>>(n, w_dev, s->fixed.p, s->w.p);
  TRY_RC(qs_tangent_alone(c));
  k_qs_fixed_rows<<<g1(n), kQsBlock, 0, c->stream>>>(n, w_dev, s->fixed.p, s->q.p);
  PD_CUDA_TRY(c, cudaMemcpyAsync(kw_dev, s->q.p, 3 * n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  return PD_OK;
}

// Tangent products of kQsMulti vectors at once (the probes of the rigid coarse
// space): the bond geometry is streamed once for all of them. p and q hold the
// vectors point-major, p[(i * kQsMulti + v) * 3 + c]; prescribed components of
// p are dropped; prescribed rows of q = p. dth [kQsMulti n] scratch.
__global__ void __launch_bounds__(kQsBlock) k_qs_dtheta_multi(int64_t n, const int64_t* __restrict__ row,
                                                              const double4* __restrict__ g,
                                                              const double4* __restrict__ ab,
                                                              const double4* __restrict__ pt,
                                                              const uint8_t* __restrict__ fixed,
                                                              const double* __restrict__ p, double* __restrict__ dth) {
  constexpr int NV = kQsMulti;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kQsTpo;
  const int lane = threadIdx.x & (kQsTpo - 1);
  const bool valid = i < n;
  double acc[NV];
  for (int v = 0; v < NV; ++v) acc[v] = 0.0;
  if (valid) {
    double pi[NV][3];
    const uint8_t fi = fixed[i];
    for (int v = 0; v < NV; ++v)
      for (int c = 0; c < 3; ++c) pi[v][c] = ((fi >> c) & 1) ? 0.0 : p[(i * NV + v) * 3 + c];
    for (int64_t b = row[i] + lane; b < row[i + 1]; b += kQsTpo) {
      const double4 gb = ld_bond(g + b);
      const int64_t j = bond_id(gb);
      const uint8_t fj = fixed[j];
      const double* pj = p + j * NV * 3;
      for (int v = 0; v < NV; ++v) {
        const double w0 = ((fj & 1) ? 0.0 : pj[3 * v]) - pi[v][0];
        const double w1 = ((fj & 2) ? 0.0 : pj[3 * v + 1]) - pi[v][1];
        const double w2 = ((fj & 4) ? 0.0 : pj[3 * v + 2]) - pi[v][2];
        acc[v] += gb.x * w0 + gb.y * w1 + gb.z * w2;
      }
    }
  }
  for (int v = 0; v < NV; ++v) acc[v] = qs_group_sum(acc[v]);
  if (valid && lane == 0) {
    const double s = 3.0 * (ab[i].y / pt[i].x);
    for (int v = 0; v < NV; ++v) dth[i * NV + v] = s * acc[v];
  }
}

__global__ void __launch_bounds__(kQsBlock) k_qs_df_multi(int64_t n, const int64_t* __restrict__ row,
                                                          const double4* __restrict__ g,
                                                          const double2* __restrict__ gc,
                                                          const double4* __restrict__ xv,
                                                          const uint8_t* __restrict__ fixed,
                                                          const double* __restrict__ p,
                                                          const double* __restrict__ dth, double* __restrict__ q) {
  constexpr int NV = kQsMulti;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kQsTpo;
  const int lane = threadIdx.x & (kQsTpo - 1);
  const bool valid = i < n;
  double d[NV][3];
  for (int v = 0; v < NV; ++v) d[v][0] = d[v][1] = d[v][2] = 0.0;
  uint8_t fi = 0;
  if (valid) {
    double pi[NV][3], ti[NV];
    fi = fixed[i];
    for (int v = 0; v < NV; ++v) {
      ti[v] = dth[i * NV + v];
      for (int c = 0; c < 3; ++c) pi[v][c] = ((fi >> c) & 1) ? 0.0 : p[(i * NV + v) * 3 + c];
    }
    for (int64_t b = row[i] + lane; b < row[i + 1]; b += kQsTpo) {
      const double4 gb = ld_bond(g + b);
      const double2 cb = gc[b];
      const int64_t j = bond_id(gb);
      const uint8_t fj = fixed[j];
      const double* pj = p + j * NV * 3;
      const double* tj = dth + j * NV;
      for (int v = 0; v < NV; ++v) {
        const double w0 = ((fj & 1) ? 0.0 : pj[3 * v]) - pi[v][0];
        const double w1 = ((fj & 2) ? 0.0 : pj[3 * v + 1]) - pi[v][1];
        const double w2 = ((fj & 4) ? 0.0 : pj[3 * v + 2]) - pi[v][2];
        const double sy = (ti[v] + tj[v]) + cb.x * (gb.x * w0 + gb.y * w1 + gb.z * w2);
        d[v][0] += sy * gb.x + cb.y * w0;
        d[v][1] += sy * gb.y + cb.y * w1;
        d[v][2] += sy * gb.z + cb.y * w2;
      }
    }
  }
  for (int v = 0; v < NV; ++v)
    for (int c = 0; c < 3; ++c) d[v][c] = qs_group_sum(d[v][c]);
  if (valid && lane < 3) {
    const int c = lane;
    const double V = xv[i].w;
    for (int v = 0; v < NV; ++v) {
      const int64_t k = (i * NV + v) * 3 + c;
      const double dv = c == 0 ? d[v][0] : (c == 1 ? d[v][1] : d[v][2]);
      q[k] = ((fi >> c) & 1) ? p[k] : -V * dv;
    }
  }
}

// q = K p for kQsMulti vectors (point-major, see k_qs_dtheta_multi) with the
// tangent prepared by qs_prepare_current; dth [kQsMulti n] scratch.
int qs_apply_K_multi(pd_ctx* c, const double* p_dev, double* q_dev, double* dth_dev) {
  QsState* s = c->qs;
  const int64_t n = c->n;
  TRY_RC(qs_geometry(c));
  k_qs_dtheta_multi<<<gt(n), kQsBlock, 0, c->stream>>>(n, c->row.p, s->geo.p, s->abq.p, c->pt.p,
                                                       s->fixed.p, p_dev, dth_dev);
  k_qs_df_multi<<<gt(n), kQsBlock, 0, c->stream>>>(n, c->row.p, s->geo.p, s->gco.p, c->xv.p, s->fixed.p,
                                                   p_dev, dth_dev, q_dev);
  PD_CUDA_TRY(c, cudaGetLastError());
  return PD_OK;
}

int qs_load_step(pd_ctx* c, double t_prev, double t_cur, const pd_qs_options* o, pd_stats* st) {
  TRY_RC(ensure_ready_internal(c));
  if (c->material_model != PD_MATERIAL_LPS) {
    c->err = "the quasi-static solve supports the LPS material model only";
    return PD_ERR_UNSUPPORTED;
  }
  if (c->phantoms) {
    c->err = "the implicit and quasi-static solves need symmetric bond families (one horizon across the blocks)";
    return PD_ERR_UNSUPPORTED;
  }
  TRY_RC(qs_alloc(c));
  QsState* s = c->qs;
  const int64_t n = c->n, m = 3 * n;
  const int precond = o->preconditioner;
  if (precond == PD_PRECOND_MPNN && !mpnn_ready(c)) {
    c->err = "the learned preconditioner is not trained (pd_mpnn_train) or loaded";
    return PD_ERR_STATE;
  }
  // prescribed dofs and their increments (DirichletIncrementBC on deltaU)
  std::vector<uint8_t> fx(n, 0);
  for (int64_t i = 0; i < n; ++i) fx[i] = c->h_bc_mask.empty() ? 0 : (uint8_t)(c->h_bc_mask[i] & 7);  // the coordinates held
  PD_CUDA_TRY(c, cudaMemcpyAsync(s->fixed.p, fx.data(), n, cudaMemcpyHostToDevice, c->stream));
  const double dt = t_cur - t_prev;
  const bool predict = o->use_predictor && st && st->steps > 0;
  // prescribed functions of x, y, z, t: their values at the two times
  const double2* fcp = nullptr;
  if (c->n_bc_expr && c->has_bc) {
    PD_CUDA_TRY(c, launch_bc_expr_at(c, t_cur, t_prev));
    fcp = c->bc_cp.p;
  }
  double l2, linf;
  // Negative tolerance: relative to the metric of this load step's start
  // without the predictor (prescribed increments only), the scale of the load
  // increment; the predicted start can sit close to the FP64 floor.
  double ref_metric = 0.0;
  if (o->newton_tolerance < 0.0 || !predict) {
    PD_CUDA_TRY(c, cudaMemsetAsync(s->du.p, 0, m * sizeof(double), c->stream));
    if (c->has_bc)
      k_qs_apply_bc<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->bc_mask.p, c->bc_a.p, c->bc_b.p, fcp, t_cur, t_prev,
                                                        c->u.p, s->du.p);
    TRY_RC(qs_residual(c, &l2, &linf));
    ref_metric = l2 + 20.0 * linf;
  }
  if (predict) {
    PD_CUDA_TRY(c, cudaMemcpyAsync(s->du.p, s->pred.p, m * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
    if (c->has_bc)
      k_qs_apply_bc<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->bc_mask.p, c->bc_a.p, c->bc_b.p, fcp, t_cur, t_prev,
                                                        c->u.p, s->du.p);
    TRY_RC(qs_residual(c, &l2, &linf));
  }
  double metric = l2 + 20.0 * linf;
  const double newton_tol = o->newton_tolerance < 0.0 ? -o->newton_tolerance * ref_metric : o->newton_tolerance;
  int newton = 0, cg_total = 0;
  int64_t coarse_builds = 0;
  double last_rel = 0.0;
  const int64_t fallbacks0 = c->qs_fallbacks;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, c->stream);
  const bool two_level =
      precond == PD_PRECOND_TWO_LEVEL || (precond == PD_PRECOND_MPNN && mpnn_coarse_cell(c) >= 0.0);
  const double cell = precond == PD_PRECOND_MPNN ? mpnn_coarse_cell(c) : o->coarse_cell;
  s->coarse_on = false;
  while (metric > newton_tol && newton < o->max_newton_iterations) {
    if (precond != PD_PRECOND_NONE) {
      k_qs_qm<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->pt.p, s->abq.p);
      k_qs_block_diag<<<gt(n), kQsBlock, 0, c->stream>>>(n, c->row.p, c->col.p, c->dmg.p, c->xv.p, s->yq.p, s->abq.p,
                                                         c->pt.p, c->hp.p, c->influence, s->fixed.p, s->dinv.p, 1);
      PD_CUDA_TRY(c, cudaGetLastError());
      if (precond == PD_PRECOND_MPNN) TRY_RC(mpnn_prepare(c, s->dinv.p));
    }
    if (two_level) {
      if (s->coarse_rebuild || !coarse_valid(c) || s->coarse_cell != std::max(0.0, cell)) {
        TRY_RC(coarse_build(c, s->yq.p, s->abq.p, s->fixed.p, std::max(0.0, cell), nullptr));
        s->coarse_cell = std::max(0.0, cell);
        s->coarse_ref_iters = -1;
        s->coarse_rebuild = false;
        ++coarse_builds;
      }
      s->coarse_on = true;
    }
    int its = 0;
    double rel = 0.0;
    int rc = qs_cg(c, precond, o->cg_relative_tolerance, o->max_cg_iterations, &its, &rel);
    cg_total += its;
    last_rel = rel;
    if (two_level) {
      // rebuild when a solve needs clearly more iterations than the first one
      // after the last build: 1.3x + 5 for the translations (a build costs a
      // few CG iterations), 2x + 10 with the rotations (a build costs ~150)
      const bool rigid = c->coarse_modes == 6;
      if (s->coarse_ref_iters < 0) s->coarse_ref_iters = its;
      else if (its > (rigid ? 2 * s->coarse_ref_iters + 10 : (13 * s->coarse_ref_iters) / 10 + 5))
        s->coarse_rebuild = true;
    }
    if (rc != PD_OK && rc != PD_ERR_NOT_CONVERGED) return rc;
    // du += alpha * x, backtracking on the convergence metric
    double alpha = 1.0, prev = metric;
    k_qs_axpy<<<g1(m), kQsBlock, 0, c->stream>>>(m, alpha, s->x.p, s->du.p);
    TRY_RC(qs_residual(c, &l2, &linf));
    metric = l2 + 20.0 * linf;
    for (int k = 0; k < 8 && !(metric < prev); ++k) {
      k_qs_axpy<<<g1(m), kQsBlock, 0, c->stream>>>(m, -0.5 * alpha, s->x.p, s->du.p);
      alpha *= 0.5;
      TRY_RC(qs_residual(c, &l2, &linf));
      metric = l2 + 20.0 * linf;
    }
    ++newton;
  }
  cudaEventRecord(e1, c->stream);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  // commit: u += du, v = du/dt (Peridigm.cpp:2858-2862); predictor for the next step
  k_qs_finish<<<g1(m), kQsBlock, 0, c->stream>>>(m, dt != 0.0 ? 1.0 / dt : 0.0, s->du.p, c->u.p, c->v.p);
  PD_CUDA_TRY(c, cudaMemcpyAsync(s->pred.p, s->du.p, m * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  PD_CUDA_TRY(c, cudaMemcpyAsync(c->f.p, s->f.p, m * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  PD_CUDA_TRY(c, cudaMemcpyAsync(c->theta.p, s->th.p, n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  c->cur = 0;
  PD_CUDA_TRY(c, launch_sync_state(c));
  PD_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  if (st) {
    st->steps += 1;
    st->newton_iterations += newton;
    st->cg_iterations += cg_total;
    st->final_residual = last_rel;
    st->preconditioner_fallbacks += c->qs_fallbacks - fallbacks0;
    st->coarse_builds += coarse_builds;
    st->device_ms += ms;
    st->bonds = c->nb_user;
  }
  if (metric > newton_tol) {
    c->err = "quasi-static Newton iteration did not reach its tolerance";
    return PD_ERR_NOT_CONVERGED;
  }
  return PD_OK;
}

// ---------------------------------------------------------------------------
// Implicit dynamics (Peridigm::executeImplicit, src/core/Peridigm.cpp:3620-4016):
// Newmark-beta steps, each solved by Newton on R = beta dt^2 (rho a - f) with
// the prescribed rows zeroed, the operator rho I + beta dt^2 K
// (computeImplicitJacobian :4319-4338, K = -d(V f)/du as in the quasi-static
// tangent) applied matrix-free, CG on it (Belos BlockCG in the reference).
// Vector updates follow the reference's Epetra Update/Scale order, without
// fused multiply-adds.
// ---------------------------------------------------------------------------
// u2 = un + dt vn + cu an, v2 = vn + cv an (:3726-3730); u = u2, a = (u - u2)
// * (1/(beta dt^2)) = 0, v = v2 + dt gamma a = v2 (:3752-3759).
__global__ void k_imp_predict(int64_t m, double dt, double cu, double cv, double* __restrict__ u,
                              double* __restrict__ v, double* __restrict__ a, double* __restrict__ u2,
                              double* __restrict__ v2) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const double un = u[k], vn = v[k], an = a[k];
  const double p = __dadd_rn(__dadd_rn(un, __dmul_rn(dt, vn)), __dmul_rn(cu, an));
  const double q = __dadd_rn(vn, __dmul_rn(cv, an));
  u2[k] = p;
  v2[k] = q;
  u[k] = p;
  a[k] = 0.0;
  v[k] = q;
}

// u += du; a = (u - u2) * (1/(beta dt^2)); v = v2 + dt gamma a (:3893-3902).
__global__ void k_imp_correct(int64_t m, double ibdt2, double dtg, const double* __restrict__ du,
                              double* __restrict__ u, const double* __restrict__ u2, double* __restrict__ a,
                              const double* __restrict__ v2, double* __restrict__ v) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const double uu = __dadd_rn(u[k], du[k]);
  const double aa = __dmul_rn(__dsub_rn(uu, u2[k]), ibdt2);
  u[k] = uu;
  a[k] = aa;
  v[k] = __dadd_rn(v2[k], __dmul_rn(dtg, aa));
}

// R = beta dt^2 (rho a - f) (:3803-3806) with the prescribed rows zeroed
// (:3810); rhs = -R for J du = -R; block partials (sum R^2, max |R|).
__global__ void k_imp_residual(int64_t n, double bdt2, const double* __restrict__ f, const double* __restrict__ a,
                               const double4* __restrict__ pt, const uint8_t* __restrict__ fixed,
                               double* __restrict__ rhs, double* __restrict__ partial) {
  __shared__ double s2[kQsBlock], sm[kQsBlock];
  double a2 = 0.0, am = 0.0;
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < 3 * n; k += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = k / 3;
    const int c = (int)(k - 3 * i);
    double r = __dmul_rn(bdt2, __dsub_rn(__dmul_rn(pt[i].w, a[k]), f[k]));
    if ((fixed[i] >> c) & 1) r = 0.0;
    rhs[k] = -r;
    a2 += r * r;
    am = fmax(am, fabs(r));
  }
  s2[threadIdx.x] = a2;
  sm[threadIdx.x] = am;
  __syncthreads();
  for (int o = kQsBlock / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      s2[threadIdx.x] += s2[threadIdx.x + o];
      sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = s2[0];
    partial[2 * blockIdx.x + 1] = sm[0];
  }
}

// Prescribed dofs at the run's start: u = a t0 + b, v = a (the rate).
__global__ void k_imp_bc_start(int64_t n, const uint8_t* __restrict__ mask, const double* __restrict__ ba,
                               const double* __restrict__ bb, double t0, double* __restrict__ u,
                               double* __restrict__ v, double* __restrict__ a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int c = 0; c < 3; ++c)
    if ((mask[i] >> c) & 1) {
      const int64_t k = 3 * i + c;
      u[k] = ba[k] * t0 + bb[k];
      v[k] = ba[k];
      a[k] = 0.0;
    }
}

// Force density at x + u (frozen bond damage) and the residual norm ||R||_2.
static int imp_residual(pd_ctx* c, double bdt2, double* norm) {
  QsState* s = c->qs;
  const int64_t n = c->n;
  k_qs_positions<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->xv.p, c->u.p, s->du.p, s->yq.p);
  PD_CUDA_TRY(c, launch_fp64_eval_at(c, s->yq.p, s->abq.p, s->th.p, s->nd.p, s->f.p));
  s->geo_dirty = true;
  k_imp_residual<<<kRedBlocks, kQsBlock, 0, c->stream>>>(n, bdt2, s->f.p, c->a.p, c->pt.p, s->fixed.p, s->r.p,
                                                         s->partial.p);
  k_qs_reduce<<<1, kQsBlock, 0, c->stream>>>(s->partial.p, kRedBlocks, 2, 1, s->scal.p + 8);
  PD_CUDA_TRY(c, cudaGetLastError());
  double h[2];
  PD_CUDA_TRY(c, cudaMemcpyAsync(h, s->scal.p + 8, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  PD_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  *norm = std::sqrt(h[0]);
  if (!std::isfinite(*norm)) {
    c->err = "NaN returned by force evaluation";
    return PD_ERR_NONFINITE;
  }
  return PD_OK;
}

int implicit_run(pd_ctx* c, double dt, double t0, int64_t nsteps, const pd_implicit_options* o, pd_stats* st) {
  TRY_RC(ensure_ready_internal(c));
  if (c->material_model != PD_MATERIAL_LPS) {
    c->err = "the implicit solve supports the LPS material model only";
    return PD_ERR_UNSUPPORTED;
  }
  if (c->n_bc_expr) {
    c->err = "prescribed displacement functions of x, y, z, t run on the explicit and quasi-static paths; give "
             "the implicit solve a*t + b";
    return PD_ERR_UNSUPPORTED;
  }
  if (c->phantoms) {
    c->err = "the implicit and quasi-static solves need symmetric bond families (one horizon across the blocks)";
    return PD_ERR_UNSUPPORTED;
  }
  TRY_RC(qs_alloc(c));
  QsState* s = c->qs;
  const int64_t n = c->n, m = 3 * n;
  PD_CUDA_TRY(c, s->v2.alloc(m));
  std::vector<uint8_t> fx(n, 0);
  for (int64_t i = 0; i < n; ++i) fx[i] = c->h_bc_mask.empty() ? 0 : (uint8_t)(c->h_bc_mask[i] & 7);  // the coordinates held
  PD_CUDA_TRY(c, cudaMemcpyAsync(s->fixed.p, fx.data(), n, cudaMemcpyHostToDevice, c->stream));
  PD_CUDA_TRY(c, cudaMemsetAsync(s->du.p, 0, m * sizeof(double), c->stream));
  if (c->has_bc)
    k_imp_bc_start<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->bc_mask.p, c->bc_a.p, c->bc_b.p, t0, c->u.p, c->v.p,
                                                      c->a.p);
  const double beta = o->beta, gamma = o->gamma;
  const double dt2 = dt * dt, bdt2 = beta * dt2, ibdt2 = 1.0 / bdt2, dtg = dt * gamma;
  const double cu = 0.5 * dt2 * (1.0 - 2.0 * beta), cv = dt * (1.0 - gamma);
  s->jk = bdt2;
  s->jm = 1.0;
  s->coarse_on = false;
  const int precond = o->preconditioner;
  int64_t newton_total = 0, cg_total = 0;
  double last_rel = 0.0;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, c->stream);
  int rc = PD_OK;
  for (int64_t step = 0; step < nsteps && rc == PD_OK; ++step) {
    k_imp_predict<<<g1(m), kQsBlock, 0, c->stream>>>(m, dt, cu, cv, c->u.p, c->v.p, c->a.p, s->pred.p, s->v2.p);
    double norm = 0.0;
    rc = imp_residual(c, bdt2, &norm);
    int it = 0;
    while (rc == PD_OK && norm > o->absolute_tolerance && it <= o->max_newton_iterations) {
      if (precond == PD_PRECOND_BLOCK_JACOBI) {
        k_qs_qm<<<g1(n), kQsBlock, 0, c->stream>>>(n, c->pt.p, s->abq.p);
        k_qs_block_diag<<<gt(n), kQsBlock, 0, c->stream>>>(n, c->row.p, c->col.p, c->dmg.p, c->xv.p, s->yq.p,
                                                           s->abq.p, c->pt.p, c->hp.p, c->influence, s->fixed.p,
                                                           s->dinv.p, 1, s->jk, s->jm);
      }
      int its = 0;
      double rel = 0.0;
      const int r2 = qs_cg_run(c, precond, o->cg_relative_tolerance, o->max_cg_iterations, &its, &rel);
      if (r2 != PD_OK && r2 != PD_ERR_NOT_CONVERGED) {  // a CG that stops short is used as it is (:3870-3872)
        rc = r2;
        break;
      }
      cg_total += its;
      last_rel = rel;
      k_imp_correct<<<g1(m), kQsBlock, 0, c->stream>>>(m, ibdt2, dtg, s->x.p, c->u.p, s->pred.p, c->a.p, s->v2.p,
                                                       c->v.p);
      rc = imp_residual(c, bdt2, &norm);
      ++it;
    }
    newton_total += it;
  }
  s->jk = 1.0;
  s->jm = 0.0;
  cudaEventRecord(e1, c->stream);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc != PD_OK) return rc;
  PD_CUDA_TRY(c, cudaMemcpyAsync(c->f.p, s->f.p, m * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  PD_CUDA_TRY(c, cudaMemcpyAsync(c->theta.p, s->th.p, n * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
  c->cur = 0;
  PD_CUDA_TRY(c, launch_sync_state(c));
  PD_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  if (st) {
    st->steps += nsteps;
    st->newton_iterations += newton_total;
    st->cg_iterations += cg_total;
    st->final_residual = last_rel;
    st->device_ms += ms;
    st->bonds = c->nb_user;
  }
  return PD_OK;
}

}  // namespace pdb
