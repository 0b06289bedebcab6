// esqs.cu -- the quasi-static ElasticState model (QuasiStaticModel<ElasticState>,
// src/model/quasistatic/QuasiStaticModel.cpp) on the GPU: force density,
// residual, the finite-difference Jacobian of assembly_jacobian_matrix_part
// (:361-454) and a BiCGSTAB solve over it.
//
// Nodes are in the handle's internal order with S doubles per node (S = 2 in
// 2-D and for 1-D meshes, whose y coordinate is zero; S = 4 in 3-D).  The
// material law uses the model dimension mdim (1, 2 or 3); components at or
// above mdim, and the components a Displacement_BC prescribes, are fixed dofs.
// A fixed dof is not an unknown: its residual entry is 0 and its Jacobian row
// and column are the identity's.
//
// Forces follow the gather form f_i = sum_j (t_ij + t_ji) M_ij omega_ij V_j of
// the reference's scatter (QuasiStaticModel.cpp:168-239, ElasticState::getBondEF,
// ElasticState.cpp:160-271); no bond breaks in the quasi-static model.
// Compiled with --fmad=false; sums run in neighbour-list order.

#include <algorithm>

#include "es_common.cuh"
#include "esqs_internal.h"
#include "fp32_common.cuh"
#include "state_io.cuh"

namespace nlm {

namespace {

__device__ __forceinline__ bool dof_fixed(uint8_t fl, int d, int mdim) {
  return d >= mdim || ((fl >> d) & 1u);
}

// Force state t for the model dimension; 1-D: alpha = E / m_i, t = alpha e
// (ElasticState.cpp:172-189).
__device__ __forceinline__ double esqs_t(const StepParams &P, int mdim, double mi, double th,
                                         double e, double Xl) {
  if (mdim == 1) {
    const double alpha = P.es_E / mi;
    return alpha * 1. * e;
  }
  return mdim == 2 ? es_t64<2>(P, mi, th, e, Xl) : es_t64<3>(P, mi, th, e, Xl);
}

// Dilatations and forces: G lanes per node (1 or 8) evaluate the bonds of a
// group of G side by side, and their terms are added in row order.  With one
// thread per node a 1,440-node plate keeps one warp in flight on 45 SMs:
// 60 + 162 us for the two kernels, 14 + 39 us with 8 lanes.

// theta_i = sum_j (c / m_i) f2 |X| e omega V_j over every bond, c = mdim, f2 =
// factor2D in 2-D (stateBasedHelperFunctions.cpp:26-83).
template <int SD, int G>
__global__ void __launch_bounds__(128)
    k_esqs_theta(const StepParams P, const DevPtrs D, int mdim, const double *u, double *theta) {
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  if (i >= P.n) return;
  const int c = threadIdx.x % G;
  const unsigned team = G == 1 ? 0u : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G);
  double xi[3], ui[3];
  ld_node<SD>(D.pos64, i, xi);
  ld_node_rw<SD>(u, i, ui);
  const double cm = (double)mdim / D.mw64[i] * (mdim == 2 ? P.es_factor2D : 1.) * 1.;
  const int64_t r0 = D.rowptr[i];
  const int len = (int)(D.rowptr[i + 1] - r0);
  double th = 0.;
  for (int kb = 0; kb < len; kb += G) {
    const int j = D.cols[r0 + min(kb + c, len - 1)];
    double xj[3], uj[3], Y[3], Xl, e;
    ld_node<SD>(D.pos64, j, xj);
    ld_node_rw<SD>(u, j, uj);
    es_geom64<SD>(xi, ui, xj, uj, Y, Xl, e);
    const double t = cm * Xl * e * es_omega(P, Xl) * D.vol64[j];
#pragma unroll
    for (int g = 0; g < G; g++) {
      const double q = G == 1 ? t : __shfl_sync(team, t, g, G);
      if (kb + g < len) th += q;
    }
  }
  if (c == 0) theta[i] = th;
}

template <int SD, int G>
__global__ void __launch_bounds__(128)
    k_esqs_force(const StepParams P, const DevPtrs D, int mdim, const double *u,
                 const double *theta, double *f) {
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  if (i >= P.n) return;
  const int c = threadIdx.x % G;
  const unsigned team = G == 1 ? 0u : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G);
  double xi[3], ui[3];
  ld_node<SD>(D.pos64, i, xi);
  ld_node_rw<SD>(u, i, ui);
  const double mi = D.mw64[i], thi = theta[i];
  const int64_t r0 = D.rowptr[i];
  const int len = (int)(D.rowptr[i + 1] - r0);
  double fi[3] = {0., 0., 0.};
  for (int kb = 0; kb < len; kb += G) {
    const int j = D.cols[r0 + min(kb + c, len - 1)];
    double xj[3], uj[3], Y[3], Xl, e;
    ld_node<SD>(D.pos64, j, xj);
    ld_node_rw<SD>(u, j, uj);
    es_geom64<SD>(xi, ui, xj, uj, Y, Xl, e);
    const double Yl = sqrt(Y[0] * Y[0] + Y[1] * Y[1] + Y[2] * Y[2]);
    const double tsum = esqs_t(P, mdim, mi, thi, e, Xl) + esqs_t(P, mdim, D.mw64[j], theta[j], e, Xl);
    const double s = tsum * es_omega(P, Xl) * D.vol64[j];
    for (int d = 0; d < SD; d++) {
      const double t = (Y[d] / Yl) * s;
#pragma unroll
      for (int g = 0; g < G; g++) {
        const double q = G == 1 ? t : __shfl_sync(team, t, g, G);
        if (kb + g < len) fi[d] = fi[d] + q;
      }
    }
  }
  if (c == 0) st_node<SD>(f, i, fi);
}

// r = f + b on free dofs, 0 on fixed ones (QuasiStaticModel::computeResidual,
// :596-646).
template <int SD>
__global__ void k_esqs_residual(int64_t n, const uint8_t *flags, int mdim, const double *f,
                                const double *b, double *r) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  constexpr int S = SD == 2 ? 2 : 4;
  const uint8_t fl = flags[i];
  for (int d = 0; d < S; d++) {
    const int64_t q = S * i + d;
    r[q] = (d < 3 && !dof_fixed(fl, d, mdim)) ? f[q] + b[q] : 0.;
  }
}

// ---- Jacobian ------------------------------------------------------------
// assembly_jacobian_matrix_part (:361-454) takes, for a row node i and each j
// in {i} U N(i), central differences of f_i with each free component rr of u_j
// moved by +-eps.  Two full force evaluations per entry cost O(len^3) bond
// evaluations per row.  Moving u_j changes only the bonds that end at j: the
// force of bond i-j at given dilatations, and the dilatations of j and of its
// neighbours, in which f_i is linear.  So the central differences are taken
// per bond, once, and a row is assembled from them, O(len^2):
//   J(i; j) = G_i (x) dtheta_i/du_j + sum_k H_ik (x) dtheta_k/du_j + A_ij
// with H_ik = dF_ik/dtheta_k, G_i = sum_k dF_ik/dtheta_i, A_ij the difference
// of F_ij, dtheta_k/du_j = B_kj for j in N(k) and -sum_j B_kj for j = k, and
// A_ii = -sum_k A_ik (a bond's extension depends on u_j - u_i only).
// Bound by latency at a few thousand rows.  40 x 36 plate, horizon 3h: a load
// step with three Jacobians took 135 ms before and 89 ms with these kernels.

// A warp per row i, a lane per bond q = (i, j): per bond B and H (MD doubles each)
// go to bond, A (MD^2, row-major) to the place of the bond's block in J, and the
// row's sums of B, g = dF_ij/dtheta_i and A, in one fixed order, to sums.  (With g
// and A in bond as well and the sums in a launch of their own, the workspace of a
// 3-D bond was 144 bytes beside the 72 of J, 48 now; same bits.)
template <int SD, int MD>
__global__ void __launch_bounds__(128)
    k_esqs_bonds(const StepParams P, const DevPtrs D, const double *u, const double *theta,
                 double eps, double *bond, double *sums, double *J) {
  constexpr int R = 2 * MD, Q = 2 * MD + MD * MD, M2 = MD * MD;
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (i >= P.n) return;
  const int lane = threadIdx.x & 31;
  double xi[3], ui[3];
  ld_node<SD>(D.pos64, i, xi);
  ld_node_rw<SD>(u, i, ui);
  const double mi = D.mw64[i], thi = theta[i];
  double sum[Q] = {};
  for (int64_t q = D.rowptr[i] + lane; q < D.rowptr[i + 1]; q += 32) {
    const int64_t j = D.cols[q];
    double xj[3], uj[3], Y[3], Xl, e;
    ld_node<SD>(D.pos64, j, xj);
    ld_node_rw<SD>(u, j, uj);
    es_geom64<SD>(xi, ui, xj, uj, Y, Xl, e);
    const double Yl = sqrt(Y[0] * Y[0] + Y[1] * Y[1] + Y[2] * Y[2]);
    const double mj = D.mw64[j], thj = theta[j];
    const double wv = es_omega(P, Xl) * D.vol64[j];
    const double cth = ((double)MD / mi) * (MD == 2 ? P.es_factor2D : 1.) * Xl * wv;
    // dt/dtheta of both ends
    double ai = 0., aj = 0.;
    if (MD == 2) {
      const double2 ci = es_coef64<2>(P, mi), cj = es_coef64<2>(P, mj);
      ai = (ci.x / 3. - ci.y) * Xl / 3.;
      aj = (cj.x / 3. - cj.y) * Xl / 3.;
    } else if (MD == 3) {
      const double2 ci = es_coef64<3>(P, mi), cj = es_coef64<3>(P, mj);
      ai = (ci.x - (P.es_ref_compat ? 0. : ci.y)) * Xl / 3.;
      aj = (cj.x - (P.es_ref_compat ? 0. : cj.y)) * Xl / 3.;
    }
    double *o = bond + R * q, *A = J + M2 * (q + i + 1);
#pragma unroll
    for (int d = 0; d < MD; d++) {
      const double f = Y[d] / Yl * wv;
      o[MD + d] = f * aj;
      sum[MD + d] += f * ai;
    }
#pragma unroll
    for (int rr = 0; rr < MD; rr++) {
      double F[2][3], E[2];
#pragma unroll
      for (int w = 0; w < 2; w++) {
        double um[3] = {uj[0], uj[1], uj[2]}, Z[3], Xm;
        um[rr] = um[rr] + (w ? -eps : eps);
        es_geom64<SD>(xi, ui, xj, um, Z, Xm, E[w]);
        const double Zl = sqrt(Z[0] * Z[0] + Z[1] * Z[1] + Z[2] * Z[2]);
        const double s =
            (esqs_t(P, MD, mi, thi, E[w], Xl) + esqs_t(P, MD, mj, thj, E[w], Xl)) * wv;
        for (int d = 0; d < 3; d++) F[w][d] = (Z[d] / Zl) * s;
      }
      const double B = cth * (E[0] - E[1]) / (2. * eps);
      o[rr] = B;
      sum[rr] += B;
#pragma unroll
      for (int ss = 0; ss < MD; ss++) {
        const double v = (F[0][ss] - F[1][ss]) / (2. * eps);
        A[ss * MD + rr] = v;
        sum[2 * MD + ss * MD + rr] += v;
      }
    }
  }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1)
#pragma unroll
    for (int d = 0; d < Q; d++) sum[d] += __shfl_xor_sync(0xffffffffu, sum[d], s);
  if (lane == 0)
    for (int d = 0; d < Q; d++) sums[Q * i + d] = sum[d];
}

// Position of the node with original id key in row k (ascending original
// ids), or -1.
__device__ __forceinline__ int row_find(const int64_t *rowptr, const int *ocols, int64_t k,
                                        int key) {
  int64_t lo = rowptr[k], hi = rowptr[k + 1];
  const int64_t end = hi, r0 = lo;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (ocols[mid] < key)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo < end && ocols[lo] == key ? (int)(lo - r0) : -1;
}

// A block of four warps per row node i: lanes over the blocks b (b = 0: i
// itself, b = 1 + k: the k-th neighbour), warps over the neighbours k whose
// dilatation u_j moves (the search of j in row k is a chain of loads: one warp
// per row took 196 us for 1,440 rows, 35 us with four).  full = 0 keeps
// the (i, rr; j, rr) entries only, as the reference does; full = 1 whole
// blocks.  Block b of row i is row-major at J[mdim^2 (rowptr[i] + i + b)], where
// k_esqs_bonds has left A; rows and columns of fixed dofs are zero.
template <int MD>
__global__ void __launch_bounds__(128)
    k_esqs_rows(const DevPtrs D, int full, const int *ocols, const double *bond,
                const double *sums, double *J) {
  constexpr int R = 2 * MD, Q = 2 * MD + MD * MD, M2 = MD * MD;
  __shared__ double part[3][M2][32];
  const int64_t i = blockIdx.x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r0 = D.rowptr[i];
  const int len = (int)(D.rowptr[i + 1] - r0);
  const double *C = sums + Q * i, *G = C + MD, *A = C + 2 * MD;
  const uint8_t fli = D.flags[i];
  for (int b0 = 0; b0 <= len; b0 += 32) {
    const int b = b0 + lane;
    const bool in = b <= len;
    const int64_t j = in && b > 0 ? (int64_t)D.cols[r0 + b - 1] : i;
    const int key = D.perm_dev[j];
    double acc[M2] = {};
    for (int k = w; in && k < len; k += 4) {
      const int64_t kn = D.cols[r0 + k];
      double dth[MD];
      if (kn == j) {
        for (int d = 0; d < MD; d++) dth[d] = -sums[Q * kn + d];
      } else {
        const int p = row_find(D.rowptr, ocols, kn, key);
        if (p < 0) continue;
        for (int d = 0; d < MD; d++) dth[d] = bond[R * (D.rowptr[kn] + p) + d];
      }
      const double *h = bond + R * (r0 + k) + MD;
      for (int ss = 0; ss < MD; ss++)
        for (int rr = 0; rr < MD; rr++) acc[ss * MD + rr] += h[ss] * dth[rr];
    }
    if (w > 0)
      for (int d = 0; d < M2; d++) part[w - 1][d][lane] = acc[d];
    __syncthreads();
    if (w == 0 && in) {
      const uint8_t flj = D.flags[j];
      double *blk = J + M2 * (r0 + i + b);
      const double *o = bond + R * (r0 + (b > 0 ? b - 1 : 0));
      for (int ss = 0; ss < MD; ss++)
        for (int rr = 0; rr < MD; rr++) {
          const int d = ss * MD + rr;
          const double own = b == 0 ? -A[d] - G[ss] * C[rr] : blk[d] + G[ss] * o[rr];
          const double v = own + acc[d] + part[0][d][lane] + part[1][d][lane] + part[2][d][lane];
          const bool on = (full || ss == rr) && !dof_fixed(fli, ss, MD) && !dof_fixed(flj, rr, MD);
          blk[d] = on ? v : 0.;
        }
    }
    __syncthreads();
  }
}

// Original column id of every directed bond.
__global__ void k_esqs_topology(int64_t n, const DevPtrs D, int *ocols) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int64_t q = D.rowptr[i]; q < D.rowptr[i + 1]; q++) ocols[q] = D.perm_dev[D.cols[q]];
}

// ---- BiCGSTAB (van der Vorst 1992) --------------------------------------------
// One iteration is two launches with every scalar on the device:
//   dir:    ends the last iteration -- omega, x += alpha p + omega s, r = s -
//           omega t -- and starts the next: beta, p = r + beta (p - omega v),
//           v = J p, partials of rhat.v
//   shadow: alpha, s = r - alpha v, t = J s, partials of s.s, t.s, t.t, rhat.s
//           and rhat.t
// r.r and rhat.r follow from shadow's sums (r = s - omega t with omega =
// t.s / t.t), which saves the third launch a separate sum over r would need,
// unless they cancel: where r.r comes out below kBiCancel s.s (a half step that
// all but solves the system; its last bits would decide on convergence) that dir
// stops after forming r and sums it, shadow passes, and the next dir goes on from
// those sums, one pair of launches more.  r,
// p and s of a neighbour are formed where the product reads them, partial sums
// are added by one warp of every block of the next launch in one fixed order
// while the others fetch their blocks of J, and a launch after convergence does
// nothing, so the host looks at the state once per graph of kBiGraph
// iterations.  A load step of the 40 x 36 plate (418 iterations): 89 ms with six
// host waits per iteration, 13.4 ms with three launches (blocks of 128, every
// thread forming the totals), 12.2 ms now.  Bound: two dependent launches, and the
// FP64 latency of the sums (2 FP64 lanes per SM), hence the small blocks.

constexpr int kBiThreads = 64;
constexpr int kBiTeam = 8;  // lanes per row of J
constexpr double kBiCancel = 0x1p-16;  // r.r by difference: good to 2^-36 or better

// Totals of N partial arrays of gridDim.x entries each, in one fixed order
// (one warp; lane 0 ends with them).
template <int N>
__device__ __forceinline__ void bi_totals(const double *part, double tot[N]) {
  const int np = (int)gridDim.x;
  for (int a = 0; a < N; a++) tot[a] = 0.;
  for (int k = threadIdx.x & 31; k < np; k += 32)
#pragma unroll
    for (int a = 0; a < N; a++) tot[a] += __ldcg(part + a * np + k);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < N; a++) tot[a] += __shfl_xor_sync(0xffffffffu, tot[a], o);
}

// Block sums of N values per thread into part[a * gridDim.x + blockIdx.x].
template <int N>
__device__ __forceinline__ void bi_partials(double v[N], double *part) {
  static_assert(kBiThreads == 64, "two warps");
  __shared__ double sh[N];
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < N; a++) v[a] += __shfl_xor_sync(0xffffffffu, v[a], o);
  if (threadIdx.x == 32)
    for (int a = 0; a < N; a++) sh[a] = v[a];
  __syncthreads();
  if (threadIdx.x == 0)
    for (int a = 0; a < N; a++) part[a * gridDim.x + blockIdx.x] = v[a] + sh[a];
}

// s = r = rhat = rhs, the other vectors 0, shadow's partials for omega = 0.
__global__ void __launch_bounds__(kBiThreads) k_bi_init(const BiArgs B, const double *rhs) {
  double sum[5] = {};
  for (int64_t q = blockIdx.x * (int64_t)kBiThreads + threadIdx.x; q < B.m;
       q += (int64_t)gridDim.x * kBiThreads) {
    const double b = rhs[q];
    B.s[q] = B.rhat[q] = b;
    // (components a row does not write stay zero)
    B.r[q] = B.x[q] = B.p[0][q] = B.p[1][q] = B.v[0][q] = B.v[1][q] = B.t[q] = 0.;
    sum[0] += b * b;
  }
  sum[3] = sum[0];
  bi_partials<5>(sum, B.part2);
  if (blockIdx.x == 0 && threadIdx.x == 0) B.sc[2] = BiScal{1., 0., 0., 0., 0., BI_RUN, 0, 0};
}

// A team's share of row i of J (block b = g, g + 8, ...): the first PF blocks
// are fetched ahead of the launch's scalars.
template <int MD>
struct BiRow {
  static constexpr int PF = MD == 3 ? 2 : 4;
  int64_t r0, i;
  int len, col[PF];
  double blk[PF][MD * MD];
  __device__ __forceinline__ int64_t column(const BiArgs &B, int b) const {
    return b == 0 ? i : (int64_t)B.cols[r0 + b - 1];
  }
  __device__ __forceinline__ void fetch(const BiArgs &B, int64_t row, int g) {
    i = row;
    r0 = B.rowptr[i];
    len = (int)(B.rowptr[i + 1] - r0);
#pragma unroll
    for (int u = 0; u < PF; u++) {
      const int b = g + u * kBiTeam;
      col[u] = b <= len ? (int)column(B, b) : -1;
#pragma unroll
      for (int d = 0; d < MD * MD; d++)
        blk[u][d] = b <= len ? __ldg(B.J + MD * MD * (r0 + i + b) + d) : 0.;
    }
  }
  // acc = J_i y with y_j from val(j, y), the same in all lanes of the team
  template <class V>
  __device__ __forceinline__ void times(const BiArgs &B, int g, V val, double acc[MD]) const {
    for (int d = 0; d < MD; d++) acc[d] = 0.;
    auto add = [&](int64_t j, const double *a) {
      double y[MD];
      val(j, y);
      for (int ss = 0; ss < MD; ss++)
        for (int rr = 0; rr < MD; rr++) acc[ss] = __fma_rn(a[ss * MD + rr], y[rr], acc[ss]);
    };
#pragma unroll
    for (int u = 0; u < PF; u++)
      if (col[u] >= 0) add(col[u], blk[u]);
    for (int b = g + PF * kBiTeam; b <= len; b += kBiTeam) {
      double a[MD * MD];
      for (int d = 0; d < MD * MD; d++) a[d] = __ldg(B.J + MD * MD * (r0 + i + b) + d);
      add(column(B, b), a);
    }
    for (int o = kBiTeam / 2; o > 0; o >>= 1)
      for (int d = 0; d < MD; d++) acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], o);
  }
};

constexpr int64_t kBiRows = kBiThreads / kBiTeam;  // rows of a block

template <int MD>
__global__ void __launch_bounds__(kBiThreads) k_bi_dir(const BiArgs B, int k) {
  constexpr int S = MD == 3 ? 4 : 2;
  __shared__ BiScal s_sc;
  const int g = threadIdx.x % kBiTeam;
  const int64_t first_row = blockIdx.x * kBiRows + threadIdx.x / kBiTeam;
  BiRow<MD> row;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  row.fetch(B, min(first_row, B.n - 1), g);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (threadIdx.x < 32) {
    BiScal sc = B.sc[2 + ((k ^ 1) & 1)];
    // the last dir launch updated x and r and summed r.r and rhat.r
    const bool summed = sc.done == BI_SUM;
    double t[5];  // s.s, t.s, t.t, rhat.s, rhat.t
    if (summed)
      bi_totals<2>(B.part3, t);
    else
      bi_totals<5>(B.part2, t);
    if (threadIdx.x == 0) {
      if (sc.done == BI_RUN || summed) {
        const double rho = sc.rho;
        bool end, cancel = false;
        if (sc.iters == 0) {
          sc.stop2 = B.tol * B.tol * t[0];
          sc.rho = t[3];
          sc.beta = sc.omega = 0.;
          end = t[0] == 0.;
        } else {
          double rr = t[0];
          bool half = false;
          if (summed) {
            sc.rho = t[1];
          } else {
            half = t[0] <= sc.stop2 || t[2] == 0.;
            sc.omega = half ? 0. : t[1] / t[2];
            rr = __fma_rn(-sc.omega, t[1], t[0]);
            cancel = !half && sc.omega != 0. && rr < kBiCancel * t[0];
            if (!cancel) sc.rho = __fma_rn(-sc.omega, t[4], t[3]);
          }
          if (!cancel) sc.beta = (sc.rho / rho) * (sc.alpha / sc.omega);
          end = half || rr <= sc.stop2 || sc.omega == 0. || sc.iters >= B.max_iters;
        }
        if (cancel) {
          sc.done = BI_SUM;
        } else {
          if (!end) {
            sc.iters++;
            end = sc.rho == 0.;  // breakdown: keep the iterate
          }
          // the solve's last x update is still due in this launch
          sc.done = end ? BI_LAST : BI_RUN;
        }
      } else {
        sc.done = BI_DONE;
      }
      sc.moved = summed;
      s_sc = sc;
      if (blockIdx.x == 0) B.sc[k & 1] = sc;
    }
  }
  __syncthreads();
  const BiScal sc = s_sc;
  if (sc.done == BI_DONE) return;
  const double *po = B.p[(k ^ 1) & 1], *vo = B.v[(k ^ 1) & 1];
  double *pn = B.p[k & 1], *vn = B.v[k & 1];
  const double bo = -sc.beta * sc.omega;
  double rv[2] = {};
  for (int64_t i0 = blockIdx.x * kBiRows; i0 < B.n; i0 += gridDim.x * kBiRows) {
    const int64_t it = i0 + threadIdx.x / kBiTeam;
    if (it != first_row) row.fetch(B, min(it, B.n - 1), g);
    const int64_t i = row.i;
    const bool own = g == 0 && it < B.n;
    if (own && !sc.moved)
      for (int d = 0; d < MD; d++) {
        const int64_t q = S * i + d;
        const double s = B.s[q], r = __fma_rn(-sc.omega, B.t[q], s);
        B.x[q] = __fma_rn(sc.omega, s, __fma_rn(sc.alpha, po[q], B.x[q]));
        B.r[q] = r;
        if (sc.done == BI_SUM) {
          // p and v for the next launch, which reads this one's slots
          pn[q] = po[q];
          vn[q] = vo[q];
          rv[0] = __fma_rn(r, r, rv[0]);
          rv[1] = __fma_rn(B.rhat[q], r, rv[1]);
        }
      }
    if (sc.done) continue;
    auto val = [&](int64_t j, double *y) {
      for (int d = 0; d < MD; d++) {
        const int64_t q = S * j + d;
        const double r = __fma_rn(-sc.omega, B.t[q], B.s[q]);
        y[d] = __fma_rn(bo, vo[q], __fma_rn(sc.beta, po[q], r));
      }
    };
    double acc[MD];
    row.times(B, g, val, acc);
    if (own) {
      const uint8_t fl = B.flags[i];
      double y[MD];
      val(i, y);
      for (int d = 0; d < MD; d++) {
        const int64_t q = S * i + d;
        const double w = dof_fixed(fl, d, MD) ? y[d] : acc[d];
        pn[q] = y[d];
        vn[q] = w;
        rv[0] = __fma_rn(B.rhat[q], w, rv[0]);
      }
    }
  }
  if (sc.done == BI_SUM)
    bi_partials<2>(rv, B.part3);
  else if (!sc.done)
    bi_partials<1>(rv, B.part1);
}

template <int MD>
__global__ void __launch_bounds__(kBiThreads) k_bi_shadow(const BiArgs B, int k) {
  constexpr int S = MD == 3 ? 4 : 2;
  __shared__ BiScal s_sc;
  const int g = threadIdx.x % kBiTeam;
  const int64_t first_row = blockIdx.x * kBiRows + threadIdx.x / kBiTeam;
  BiRow<MD> row;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  row.fetch(B, min(first_row, B.n - 1), g);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (threadIdx.x < 32) {
    BiScal sc = B.sc[k & 1];
    double t[1];
    bi_totals<1>(B.part1, t);
    if (threadIdx.x == 0) {
      if (!sc.done) {
        if (t[0] == 0.)
          sc.done = BI_DONE;  // breakdown: keep the iterate
        else
          sc.alpha = sc.rho / t[0];
      }
      s_sc = sc;
      if (blockIdx.x == 0) B.sc[2 + (k & 1)] = sc;
    }
  }
  __syncthreads();
  const BiScal sc = s_sc;
  if (sc.done) return;
  const double *v = B.v[k & 1];
  double sums[5] = {};
  for (int64_t i0 = blockIdx.x * kBiRows; i0 < B.n; i0 += gridDim.x * kBiRows) {
    const int64_t it = i0 + threadIdx.x / kBiTeam;
    if (it != first_row) row.fetch(B, min(it, B.n - 1), g);
    const int64_t i = row.i;
    auto val = [&](int64_t j, double *y) {
      for (int d = 0; d < MD; d++) y[d] = __fma_rn(-sc.alpha, v[S * j + d], B.r[S * j + d]);
    };
    double acc[MD];
    row.times(B, g, val, acc);
    if (g == 0 && it < B.n) {
      const uint8_t fl = B.flags[i];
      double y[MD];
      val(i, y);
      for (int d = 0; d < MD; d++) {
        const int64_t q = S * i + d;
        const double t = dof_fixed(fl, d, MD) ? y[d] : acc[d], h = B.rhat[q];
        B.s[q] = y[d];
        B.t[q] = t;
        sums[0] = __fma_rn(y[d], y[d], sums[0]);
        sums[1] = __fma_rn(t, y[d], sums[1]);
        sums[2] = __fma_rn(t, t, sums[2]);
        sums[3] = __fma_rn(h, y[d], sums[3]);
        sums[4] = __fma_rn(h, t, sums[4]);
      }
    }
  }
  bi_partials<5>(sums, B.part2);
}

// out = a x + b y + c z (any of y, z may be NULL).
__global__ void k_lin3(int64_t m, double a, const double *x, double b, const double *y, double c,
                       const double *z, double *out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= m) return;
  double v = a * x[q];
  if (y) v = v + b * y[q];
  if (z) v = v + c * z[q];
  out[q] = v;
}

__global__ void k_esqs_dot(int64_t m, const double *a, const double *b, double *part) {
  __shared__ double sh[256];
  double s = 0.;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < m;
       q += (int64_t)gridDim.x * blockDim.x)
    s += a[q] * b[q];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = 128; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void k_esqs_sum(const double *part, int nparts, double *out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double s = 0.;
  for (int k = 0; k < nparts; k++) s += part[k];
  *out = s;
}

unsigned blocks_of(int64_t m, int bs) { return (unsigned)((m + bs - 1) / bs); }

}  // namespace

cudaError_t esqs_force(const StepParams &P, const DevPtrs &D, int S, int mdim, const double *u,
                       double *theta, double *f, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  // teams below 16384 nodes, where one thread per node leaves SMs idle: us per
  // evaluation with one / eight lanes, horizon 3h -- 2-D 1,440 nodes 294 / 84, 6,400:
  // 301 / 158, 10,000: 305 / 233, 16,384: 306 / 335, 62,500: 946 / 1061; 3-D 1,728:
  // 995 / 196, 15,625: 1032 / 975, 32,768: 1745 / 1764
  const int G = P.n < 16384 ? 8 : 1;
  const unsigned g = blocks_of(P.n * G, 128);
  (S == 2 ? (G == 1 ? k_esqs_theta<2, 1> : k_esqs_theta<2, 8>)
          : (G == 1 ? k_esqs_theta<3, 1> : k_esqs_theta<3, 8>))<<<g, 128, 0, s>>>(P, D, mdim, u,
                                                                                 theta);
  (S == 2 ? (G == 1 ? k_esqs_force<2, 1> : k_esqs_force<2, 8>)
          : (G == 1 ? k_esqs_force<3, 1> : k_esqs_force<3, 8>))<<<g, 128, 0, s>>>(P, D, mdim, u,
                                                                                 theta, f);
  return cudaGetLastError();
}

cudaError_t esqs_residual(const StepParams &P, const DevPtrs &D, int S, int mdim,
                          const double *f, const double *b, double *r, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  const unsigned g = blocks_of(P.n, 256);
  if (S == 2)
    k_esqs_residual<2><<<g, 256, 0, s>>>(P.n, D.flags, mdim, f, b, r);
  else
    k_esqs_residual<3><<<g, 256, 0, s>>>(P.n, D.flags, mdim, f, b, r);
  return cudaGetLastError();
}

cudaError_t esqs_topology(const StepParams &P, const DevPtrs &D, int *ocols, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  k_esqs_topology<<<blocks_of(P.n, 128), 128, 0, s>>>(P.n, D, ocols);
  return cudaGetLastError();
}

cudaError_t esqs_jacobian(const StepParams &P, const DevPtrs &D, int S, int mdim, int full,
                          const double *u, const double *theta, double eps, const int *ocols,
                          double *bond, double *sums, double *J, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  // (a mesh of 1 or 2 dimensions is stored as a 2-D one)
  (mdim == 3   ? k_esqs_bonds<3, 3>
   : mdim == 2 ? k_esqs_bonds<2, 2>
               : k_esqs_bonds<2, 1>)<<<blocks_of(32 * P.n, 128), 128, 0, s>>>(P, D, u, theta, eps,
                                                                              bond, sums, J);
  (mdim == 1   ? k_esqs_rows<1>
   : mdim == 2 ? k_esqs_rows<2>
               : k_esqs_rows<3>)<<<(unsigned)P.n, 128, 0, s>>>(D, full, ocols, bond, sums, J);
  return cudaGetLastError();
}

int esqs_bicgstab_blocks(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(kBiParts, (n + kBiRows - 1) / kBiRows));
}

// kBiGraph iterations as one CUDA graph (iteration parities 1, 0, 1, ...).
cudaError_t esqs_bicgstab_graph(const BiArgs &B, int mdim, cudaGraphExec_t *out, cudaStream_t s) {
  auto dir = mdim == 1 ? k_bi_dir<1> : mdim == 2 ? k_bi_dir<2> : k_bi_dir<3>;
  auto shadow = mdim == 1 ? k_bi_shadow<1> : mdim == 2 ? k_bi_shadow<2> : k_bi_shadow<3>;
  cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) return e;
  for (int k = 1; k <= kBiGraph && e == cudaSuccess; k++) {
    e = launch_pdl(dir, B.blocks, kBiThreads, 0, s, k > 1, B, k & 1);
    if (e == cudaSuccess) e = launch_pdl(shadow, B.blocks, kBiThreads, 0, s, true, B, k & 1);
  }
  cudaGraph_t g = nullptr;
  const cudaError_t ec = cudaStreamEndCapture(s, &g);
  if (e == cudaSuccess) e = ec;
  if (e == cudaSuccess) e = cudaGraphInstantiate(out, g, 0);
  if (g) cudaGraphDestroy(g);
  return e;
}

cudaError_t esqs_bicgstab(const BiArgs &B, cudaGraphExec_t graph, const double *rhs, int *iters,
                          cudaStream_t s) {
  k_bi_init<<<B.blocks, kBiThreads, 0, s>>>(B, rhs);
  cudaError_t e = cudaGetLastError();
  BiScal st{};
  // max_iters ends it on the device
  while (e == cudaSuccess && (st.done == BI_RUN || st.done == BI_SUM)) {
    e = cudaGraphLaunch(graph, s);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(&st, B.sc + 2, sizeof(st), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  *iters = st.iters;
  return e;
}

cudaError_t esqs_lin3(int64_t m, double a, const double *x, double b, const double *y, double c,
                      const double *z, double *out, cudaStream_t s) {
  if (m == 0) return cudaSuccess;
  k_lin3<<<blocks_of(m, 256), 256, 0, s>>>(m, a, x, b, y, c, z, out);
  return cudaGetLastError();
}

cudaError_t esqs_dot(int64_t m, const double *a, const double *b, double *part, double *out,
                     cudaStream_t s) {
  const int nparts = (int)std::min<int64_t>(kEsqsDotParts, std::max<int64_t>(1, (m + 255) / 256));
  k_esqs_dot<<<nparts, 256, 0, s>>>(m, a, b, part);
  k_esqs_sum<<<1, 32, 0, s>>>(part, nparts, out);
  return cudaGetLastError();
}

}  // namespace nlm
