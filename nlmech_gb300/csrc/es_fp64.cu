// es_fp64.cu -- ElasticState explicit step, FP64 plain (two passes).
//
// Pass 1 (k_es_dil64): per node the bond extensions e_ij = |Y_ij| - |X_ij|
// (src/util/stateBasedHelperFunctions.cpp:47), the irreversible break test
// e_ij / |X_ij| > s_c, and the dilatation over intact bonds
//   theta_i = sum_j (c / m_i) f2 |X| e omega_ij V_j   (c = 2 in 2-D, 3 in 3-D;
//   f2 = factor2D in 2-D) as in stateBasedHelperFunctions.cpp:50-79.
// Pass 2 (k_es_force64): the gather form of the reference's half-force
// scatter (QuasiStaticModel.cpp:168-239 with ElasticState::getBondEF,
// ElasticState.cpp:160-271):
//   f_i = sum_j (t_ij + t_ji) M_ij omega_ij V_j,   M = Y / |Y|,
// followed by the integrator epilogue shared with RNPBond.
// Compiled with --fmad=false; sums run in neighbour-list order.

#include <type_traits>

#include "es_common.cuh"
#include "fd_internal.h"
#include "state_io.cuh"

namespace nlm {

// Weighted volume m_i = sum_j |X|^2 omega V_j (volumeCorrection.cpp:48-67).
template <int DIM>
__global__ void k_es_mw(const StepParams P, const DevPtrs D, double *mw) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  double xi[3];
  ld_node<DIM>(D.pos64, i, xi);
  double tmp = 0.;
  for (int64_t k = D.rowptr[i]; k < D.rowptr[i + 1]; k++) {
    const int j = D.cols[k];
    double xj[3];
    ld_node<DIM>(D.pos64, j, xj);
    const double X0 = xj[0] - xi[0], X1 = xj[1] - xi[1], X2 = xj[2] - xi[2];
    const double Xl = sqrt(X0 * X0 + X1 * X1 + X2 * X2);
    tmp += (Xl * Xl * es_omega(P, Xl) * D.vol64[j]);
  }
  mw[i] = tmp;
}

template <int DIM>
__global__ void __launch_bounds__(128)
    k_es_dil64(const StepParams P, const DevPtrs D, const StepArgs A) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const double *ucur = D.u64[A.cur];
  double xi[3], ui[3];
  ld_node<DIM>(D.pos64, i, xi);
  ld_node<DIM>(ucur, i, ui);
  const int *colp = D.sell_cols + D.sell_ptr[i >> 5] + 4 * (i & 31);
  const int len = D.rowlen[i];
  const double mi = D.mw64[i];
  const double c = DIM == 2 ? 2. : 3.;
  const double fac = DIM == 2 ? P.es_factor2D : 1.;
  double th = 0.;
  uint32_t word = 0;
  bool dirty = false;
  int chunk = 0;
  for (int k = 0; k < len; k++) {
    if ((k & 31) == 0) {
      if (dirty) D.bits[(int64_t)chunk * P.npad + i] = word;
      chunk = k >> 5;
      word = D.bits[(int64_t)chunk * P.npad + i];
      dirty = false;
    }
    const int j = __ldg(colp + (k >> 2) * 128 + (k & 3));
    double xj[3], uj[3], Y[3], Xl, e;
    ld_node<DIM>(D.pos64, j, xj);
    ld_node<DIM>(ucur, j, uj);
    es_geom64<DIM>(xi, ui, xj, uj, Y, Xl, e);
    bool fs = (word >> (k & 31)) & 1u;
    if (P.es_sc > 0. && !fs && dGT(e / Xl, P.es_sc)) {
      fs = true;
      word |= 1u << (k & 31);
      dirty = true;
    }
    if (fs) continue;
    th += (c / mi) * fac * 1. * Xl * e * es_omega(P, Xl) * D.vol64[j];
  }
  if (dirty) D.bits[(int64_t)chunk * P.npad + i] = word;
  D.theta64[i] = th;
}

template <int DIM, int SCHEME>
__global__ void __launch_bounds__(128)
    k_es_force64(const StepParams P, const DevPtrs D, const StepArgs A) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  const double *ucur = D.u64[A.cur];
  double xi[3], ui[3];
  ld_node<DIM>(D.pos64, i, xi);
  ld_node<DIM>(ucur, i, ui);
  const uint8_t fl = D.flags[i];
  const int *colp = D.sell_cols + D.sell_ptr[i >> 5] + 4 * (i & 31);
  const int len = D.rowlen[i];
  const double mi = D.mw64[i], thi = D.theta64[i];
  double fi[3] = {0., 0., 0.};
  uint32_t word = 0;
  for (int k = 0; k < len; k++) {
    if ((k & 31) == 0) word = D.bits[(int64_t)(k >> 5) * P.npad + i];
    if ((word >> (k & 31)) & 1u) continue;
    const int j = __ldg(colp + (k >> 2) * 128 + (k & 3));
    double xj[3], uj[3], Y[3], Xl, e;
    ld_node<DIM>(D.pos64, j, xj);
    ld_node<DIM>(ucur, j, uj);
    es_geom64<DIM>(xi, ui, xj, uj, Y, Xl, e);
    const double Yl = sqrt(Y[0] * Y[0] + Y[1] * Y[1] + Y[2] * Y[2]);
    const double tsum =
        es_t64<DIM>(P, mi, thi, e, Xl) + es_t64<DIM>(P, D.mw64[j], D.theta64[j], e, Xl);
    const double s = tsum * es_omega(P, Xl) * D.vol64[j];
    fi[0] = fi[0] + (Y[0] / Yl) * s;
    fi[1] = fi[1] + (Y[1] / Yl) * s;
    if (DIM == 3) fi[2] = fi[2] + (Y[2] / Yl) * s;
  }
  if (A.first)
    integrate_node64<DIM, SCHEME, true>(P, D, A, i, fl, ui, fi);
  else
    integrate_node64<DIM, SCHEME, false>(P, D, A, i, fl, ui, fi);
}

// ---- the two passes over the FP64 bond store ----------------------------------
// As in fd_fp64.cu the FP64 pipe is the bound (k_es_dil64 + k_es_force64: about
// 290 FP64 instructions per bond).  |X|, omega and V_j come from the store,
// the material coefficients are per node, y = x + u is formed once per node,
// |Y| is handed from pass 1 to pass 2, divisions by 3 and by |Y| take three
// operations each (div_by), and the break test is an integer comparison with
// a bound below the extension at s_c.  The remaining operations are those of
// k_es_dil64 and k_es_force64 in their order: the same bits.  31 x 29 x 27
// block: 1596 us per step with those kernels, 371 us here (the FP64 pipe 79 and
// 84 % busy, 80 instructions per bond); 60^3 cube: 3165 us.

template <int DIM>
__global__ void k_es_store64(const StepParams P, const DevPtrs D, double2 *bx, double *bv, int *bt,
                             double2 *nc) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  double xi[3];
  ld_node<DIM>(D.pos64, i, xi);
  const int64_t base = D.sell_ptr[i >> 5];
  const int lane = (int)(i & 31), len = D.rowlen[i];
  const double mi = D.mw64[i];
  nc[i] = es_coef64<DIM>(P, mi);
  for (int k = 0; k < len; k++) {
    const int j = D.sell_cols[base + 4 * lane + (k >> 2) * 128 + (k & 3)];
    const int64_t q = base + 32 * (int64_t)k + lane;
    double xj[3], X[3];
    ld_node<DIM>(D.pos64, j, xj);
    for (int d = 0; d < 3; d++) X[d] = xj[d] - xi[d];
    const double Xl = sqrt(X[0] * X[0] + X[1] * X[1] + X[2] * X[2]);
    bx[q] = make_double2(Xl, es_omega(P, Xl));
    bv[q] = D.vol64[j];
    // e / |X| > s_c (1 + 1e-5 ...) needs e above this bound's high word
    const double lim = Xl * P.es_sc * (1. - 1e-6);
    bt[q] = P.es_sc > 0. ? max(0, min(0x7ff00000, __double2hiint(lim))) : 0x7ff00001;
  }
}

template <int DIM>
__global__ void k_es_y64(const StepParams P, const DevPtrs D, const StepArgs A) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  double x[3], u[3];
  ld_node<DIM>(D.pos64, i, x);
  ld_node<DIM>(D.u64[A.cur], i, u);
  for (int d = 0; d < 3; d++) x[d] = x[d] + u[d];
  st_node<DIM>(D.es64_y, i, x);
}

// G lanes per node and U bonds of each lane side by side, as in k_rnp64_bond.
template <int DIM, int G>
__global__ void __launch_bounds__(128) k_es_dil64_bond(const StepParams P, const DevPtrs D) {
  constexpr int U = G == 16 ? 1 : 2, W = G * U;
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  if (i >= P.n) return;
  const int c = threadIdx.x % G;
  const unsigned team = G == 1 ? 0u : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G);
  double yi[3];
  ld_node<DIM>(D.es64_y, i, yi);
  const int64_t base = D.sell_ptr[i >> 5];
  const int lane = (int)(i & 31), len = D.rowlen[i];
  const int *colp = D.sell_cols + base + 4 * lane;
  const double a = ((DIM == 2 ? 2. : 3.) / D.mw64[i]) * (DIM == 2 ? P.es_factor2D : 1.) * 1.;
  double th = 0.;
  uint32_t word = 0;
  for (int kb = 0; kb < len; kb += W) {
    if ((kb & 31) == 0) word = D.bits[(int64_t)(kb >> 5) * P.npad + i];
    double t[U];
    uint32_t add = 0, cut = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = min(kb + u * G + c, len - 1);
      const int64_t q = base + 32 * (int64_t)k + lane;
      const int j = __ldg(colp + (k >> 2) * 128 + (k & 3));
      double yj[3], Y[3];
      ld_node<DIM>(D.es64_y, j, yj);
      const double2 x = ld_once(D.es64_x + q);
      const double vj = ld_once(D.es64_v + q);
      const int thr = ld_once(D.es64_thr + q);
      for (int d = 0; d < DIM; d++) Y[d] = yj[d] - yi[d];
      double qq = Y[0] * Y[0] + Y[1] * Y[1];
      if (DIM == 3) qq = qq + Y[2] * Y[2];
      const double Yl = sqrt(qq), e = Yl - x.x;
      const bool in = kb + u * G + c < len;
      if (in) D.es64_yl[q] = Yl;
      const int b = (kb & 31) + u * G + c;
      bool fs = (word >> b) & 1u;
      // a NaN e (high word at least 0x7ff80000, or negative) breaks nothing
      if (__double2hiint(e) >= thr && !fs && in && dGT(e / x.x, P.es_sc)) {
        fs = true;
        cut |= 1u << b;
      }
      if (in && !fs) add |= 1u << u;
      t[u] = a * x.x * e * x.y * vj;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int g = 0; g < G; g++) {
        const uint32_t ad = G == 1 ? add : __shfl_sync(team, add, g, G);
        const double q = G == 1 ? t[u] : __shfl_sync(team, t[u], g, G);
        if (ad >> u & 1u) th += q;
      }
    if (G > 1)
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) cut |= __shfl_xor_sync(team, cut, o, G);
    if (cut) {
      word |= cut;
      if (c == 0) D.bits[(int64_t)(kb >> 5) * P.npad + i] = word;
    }
  }
  if (c == 0) D.theta64[i] = th;
}

// t of one side of a bond from its node's coefficients (es_t64).
template <int DIM>
__device__ __forceinline__ double es_t64_coef(const double2 c, double theta, double e, double Xl,
                                              double third, bool compat) {
  const double e_s = div_by(theta * Xl, 3., third);
  if (DIM == 2) {
    const double t_s = div_by(c.x * e_s, 3., third);
    return t_s + c.y * (e - e_s);
  }
  return c.x * e_s + c.y * (compat ? 0. : e - e_s);
}

template <int DIM, int SCHEME, int G>
__global__ void __launch_bounds__(128)
    k_es_force64_bond(const StepParams P, const DevPtrs D, const StepArgs A) {
  constexpr int U = G == 16 ? 1 : 2, W = G * U;
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  if (i >= P.n) return;
  const int c = threadIdx.x % G;
  const unsigned team = G == 1 ? 0u : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G);
  double yi[3];
  ld_node<DIM>(D.es64_y, i, yi);
  const int64_t base = D.sell_ptr[i >> 5];
  const int lane = (int)(i & 31), len = D.rowlen[i];
  const int *colp = D.sell_cols + base + 4 * lane;
  const double2 ci = D.es64_c[i];
  const double thi = D.theta64[i], third = 1. / 3.;
  const bool compat = P.es_ref_compat;
  double fi[3] = {0., 0., 0.};
  uint32_t word = 0;
  for (int kb = 0; kb < len; kb += W) {
    if ((kb & 31) == 0) word = D.bits[(int64_t)(kb >> 5) * P.npad + i];
    double p[U][DIM];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int k = min(kb + u * G + c, len - 1);
      const int64_t q = base + 32 * (int64_t)k + lane;
      const int j = __ldg(colp + (k >> 2) * 128 + (k & 3));
      const double2 x = ld_once(D.es64_x + q);
      const double vj = ld_once(D.es64_v + q);
      const double Yl = ld_once(D.es64_yl + q);
      const double2 cj = __ldg(D.es64_c + j);
      const double thj = __ldg(D.theta64 + j);
      double yj[3];
      ld_node<DIM>(D.es64_y, j, yj);
      const double e = Yl - x.x;
      const double tsum = es_t64_coef<DIM>(ci, thi, e, x.x, third, compat) +
                          es_t64_coef<DIM>(cj, thj, e, x.x, third, compat);
      const double s = tsum * x.y * vj;
      const double ry = __drcp_rn(Yl);
      for (int d = 0; d < DIM; d++) p[u][d] = div_by(yj[d] - yi[d], Yl, ry) * s;
    }
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int g = 0; g < G; g++) {
        double q[DIM];
#pragma unroll
        for (int d = 0; d < DIM; d++)
          q[d] = G == 1 ? p[u][d] : __shfl_sync(team, p[u][d], g, G);
        const int k = u * G + g;
        if (kb + k < len && !((word >> ((kb & 31) + k)) & 1u))
#pragma unroll
          for (int d = 0; d < DIM; d++) fi[d] = fi[d] + q[d];
      }
  }
  if (c) return;
  double ui[3];
  ld_node<DIM>(D.u64[A.cur], i, ui);
  const uint8_t fl = D.flags[i];
  if (A.first)
    integrate_node64<DIM, SCHEME, true>(P, D, A, i, fl, ui, fi);
  else
    integrate_node64<DIM, SCHEME, false>(P, D, A, i, fl, ui, fi);
}

cudaError_t launch_es_store64(const StepParams &P, const DevPtrs &D, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  const unsigned g = (unsigned)((P.n + 127) / 128);
  (P.dim == 2 ? k_es_store64<2> : k_es_store64<3>)<<<g, 128, 0, s>>>(
      P, D, const_cast<double2 *>(D.es64_x), const_cast<double *>(D.es64_v),
      const_cast<int *>(D.es64_thr), const_cast<double2 *>(D.es64_c));
  return cudaGetLastError();
}

template <int DIM>
static cudaError_t es64(const StepParams &P, const DevPtrs &D, const StepArgs &a, cudaStream_t s) {
  const unsigned g = (unsigned)((P.n + 127) / 128);
  if (D.es64_x) {
    const int G = team64(P.n);
    const unsigned gg = (unsigned)((P.n * G + kTeamBlock - 1) / kTeamBlock);
    const bool vv = P.scheme == NLM_VELOCITY_VERLET;
    k_es_y64<DIM><<<g, 128, 0, s>>>(P, D, a);
    auto run = [&](auto team) {
      constexpr int N = decltype(team)::value;
      k_es_dil64_bond<DIM, N><<<gg, kTeamBlock, 0, s>>>(P, D);
      (vv ? k_es_force64_bond<DIM, NLM_VELOCITY_VERLET, N>
          : k_es_force64_bond<DIM, NLM_CENTRAL_DIFFERENCE, N>)<<<gg, kTeamBlock, 0, s>>>(P, D, a);
    };
    if (G == 1)
      run(std::integral_constant<int, 1>{});
    else if (G == 2)
      run(std::integral_constant<int, 2>{});
    else if (G == 4)
      run(std::integral_constant<int, 4>{});
    else
      run(std::integral_constant<int, 16>{});
    return cudaGetLastError();
  }
  k_es_dil64<DIM><<<g, 128, 0, s>>>(P, D, a);
  if (P.scheme == NLM_VELOCITY_VERLET)
    k_es_force64<DIM, NLM_VELOCITY_VERLET><<<g, 128, 0, s>>>(P, D, a);
  else
    k_es_force64<DIM, NLM_CENTRAL_DIFFERENCE><<<g, 128, 0, s>>>(P, D, a);
  return cudaGetLastError();
}

cudaError_t launch_es_step_fp64(const StepParams &P, const DevPtrs &D, const StepArgs &a, int decomp, cudaStream_t s) {
  (void)decomp;
  if (P.n == 0) return cudaSuccess;
  return P.dim == 2 ? es64<2>(P, D, a, s) : es64<3>(P, D, a, s);
}

cudaError_t launch_es_setup(const StepParams &P, const DevPtrs &D, double *mw, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  const unsigned g = (unsigned)((P.n + 127) / 128);
  if (P.dim == 2)
    k_es_mw<2><<<g, 128, 0, s>>>(P, D, mw);
  else
    k_es_mw<3><<<g, 128, 0, s>>>(P, D, mw);
  return cudaGetLastError();
}

}  // namespace nlm
