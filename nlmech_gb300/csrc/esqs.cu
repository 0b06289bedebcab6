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

// Dilatation theta_i (stateBasedHelperFunctions.cpp:26-83, every bond):
// theta_i = sum_j (c / m_i) f2 |X| e omega V_j, c = mdim, f2 = factor2D in 2-D.
template <int SD>
__device__ double theta_node(const StepParams &P, const DevPtrs &D, int mdim, const double *u,
                             int64_t i) {
  double xi[3], ui[3];
  ld_node<SD>(D.pos64, i, xi);
  ld_node_rw<SD>(u, i, ui);
  const double mi = D.mw64[i];
  const double c = (double)mdim;
  double th = 0.;
  for (int64_t k = D.rowptr[i]; k < D.rowptr[i + 1]; k++) {
    const int j = D.cols[k];
    double xj[3], uj[3], Y[3], Xl, e;
    ld_node<SD>(D.pos64, j, xj);
    ld_node_rw<SD>(u, j, uj);
    es_geom64<SD>(xi, ui, xj, uj, Y, Xl, e);
    if (mdim == 2)
      th += (c / mi) * P.es_factor2D * 1. * Xl * e * es_omega(P, Xl) * D.vol64[j];
    else
      th += (c / mi) * 1. * Xl * e * es_omega(P, Xl) * D.vol64[j];
  }
  return th;
}

template <int SD>
__global__ void k_esqs_theta(const StepParams P, const DevPtrs D, int mdim, const double *u,
                             double *theta) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  theta[i] = theta_node<SD>(P, D, mdim, u, i);
}

template <int SD>
__global__ void k_esqs_force(const StepParams P, const DevPtrs D, int mdim, const double *u,
                             const double *theta, double *f) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  double xi[3], ui[3];
  ld_node<SD>(D.pos64, i, xi);
  ld_node_rw<SD>(u, i, ui);
  const double mi = D.mw64[i], thi = theta[i];
  double fi[3] = {0., 0., 0.};
  for (int64_t k = D.rowptr[i]; k < D.rowptr[i + 1]; k++) {
    const int j = D.cols[k];
    double xj[3], uj[3], Y[3], Xl, e;
    ld_node<SD>(D.pos64, j, xj);
    ld_node_rw<SD>(u, j, uj);
    es_geom64<SD>(xi, ui, xj, uj, Y, Xl, e);
    const double Yl = sqrt(Y[0] * Y[0] + Y[1] * Y[1] + Y[2] * Y[2]);
    const double tsum = esqs_t(P, mdim, mi, thi, e, Xl) + esqs_t(P, mdim, D.mw64[j], theta[j], e, Xl);
    const double s = tsum * es_omega(P, Xl) * D.vol64[j];
    for (int d = 0; d < 3; d++) fi[d] = fi[d] + (Y[d] / Yl) * s;
  }
  st_node<SD>(f, i, fi);
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

// One thread per directed bond q = (i, j), mdim <= 3 components; per bond
// B (mdim), H (mdim), g = dF_ij/dtheta_i (mdim) and A (mdim^2, row-major).
template <int SD>
__global__ void k_esqs_bonds(const StepParams P, const DevPtrs D, int mdim, const int *rows,
                             int64_t nnz, const double *u, const double *theta, double eps,
                             double *out) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= nnz) return;
  const int64_t i = rows[q], j = D.cols[q];
  double xi[3], ui[3], xj[3], uj[3], Y[3], Xl, e;
  ld_node<SD>(D.pos64, i, xi);
  ld_node_rw<SD>(u, i, ui);
  ld_node<SD>(D.pos64, j, xj);
  ld_node_rw<SD>(u, j, uj);
  es_geom64<SD>(xi, ui, xj, uj, Y, Xl, e);
  const double Yl = sqrt(Y[0] * Y[0] + Y[1] * Y[1] + Y[2] * Y[2]);
  const double mi = D.mw64[i], mj = D.mw64[j], thi = theta[i], thj = theta[j];
  const double wv = es_omega(P, Xl) * D.vol64[j];
  const double cth = ((double)mdim / mi) * (mdim == 2 ? P.es_factor2D : 1.) * Xl * wv;
  // dt/dtheta of both ends
  double ai = 0., aj = 0.;
  if (mdim == 2) {
    const double2 ci = es_coef64<2>(P, mi), cj = es_coef64<2>(P, mj);
    ai = (ci.x / 3. - ci.y) * Xl / 3.;
    aj = (cj.x / 3. - cj.y) * Xl / 3.;
  } else if (mdim == 3) {
    const double2 ci = es_coef64<3>(P, mi), cj = es_coef64<3>(P, mj);
    ai = (ci.x - (P.es_ref_compat ? 0. : ci.y)) * Xl / 3.;
    aj = (cj.x - (P.es_ref_compat ? 0. : cj.y)) * Xl / 3.;
  }
  double *o = out + (int64_t)(3 * mdim + mdim * mdim) * q;
  for (int d = 0; d < mdim; d++) {
    const double f = Y[d] / Yl * wv;
    o[mdim + d] = f * aj;
    o[2 * mdim + d] = f * ai;
  }
  for (int rr = 0; rr < mdim; rr++) {
    double F[2][3], E[2];
    for (int w = 0; w < 2; w++) {
      double um[3] = {uj[0], uj[1], uj[2]}, Z[3], Xm;
      um[rr] = um[rr] + (w ? -eps : eps);
      es_geom64<SD>(xi, ui, xj, um, Z, Xm, E[w]);
      const double Zl = sqrt(Z[0] * Z[0] + Z[1] * Z[1] + Z[2] * Z[2]);
      const double s =
          (esqs_t(P, mdim, mi, thi, E[w], Xl) + esqs_t(P, mdim, mj, thj, E[w], Xl)) * wv;
      for (int d = 0; d < 3; d++) F[w][d] = (Z[d] / Zl) * s;
    }
    o[rr] = cth * (E[0] - E[1]) / (2. * eps);
    for (int ss = 0; ss < mdim; ss++)
      o[3 * mdim + ss * mdim + rr] = (F[0][ss] - F[1][ss]) / (2. * eps);
  }
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

// A warp per row node i, its lanes over the blocks b (b = 0: i itself, b = 1 +
// k: the k-th neighbour).  full = 0 keeps the (i, rr; j, rr) entries only, as
// the reference does; full = 1 whole blocks.  Block b of row i is row-major at
// J[mdim^2 (rowptr[i] + i + b)]; rows and columns of fixed dofs are zero.
template <int MD>
__global__ void __launch_bounds__(128)
    k_esqs_rows(int64_t n, const DevPtrs D, int full, const int *ocols, const double *bond,
                double *J) {
  constexpr int R = 3 * MD + MD * MD;
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;
  const int lane = threadIdx.x & 31;
  const int64_t r0 = D.rowptr[i];
  const int len = (int)(D.rowptr[i + 1] - r0);
  // sums over the row, in one fixed order
  double G[MD] = {}, C[MD] = {}, A[MD * MD] = {};
  for (int k = lane; k < len; k += 32) {
    const double *o = bond + R * (r0 + k);
    for (int d = 0; d < MD; d++) {
      C[d] += o[d];
      G[d] += o[2 * MD + d];
    }
    for (int d = 0; d < MD * MD; d++) A[d] += o[3 * MD + d];
  }
  for (int s = 16; s > 0; s >>= 1) {
    for (int d = 0; d < MD; d++) {
      C[d] += __shfl_xor_sync(0xffffffffu, C[d], s);
      G[d] += __shfl_xor_sync(0xffffffffu, G[d], s);
    }
    for (int d = 0; d < MD * MD; d++) A[d] += __shfl_xor_sync(0xffffffffu, A[d], s);
  }
  const uint8_t fli = D.flags[i];
  for (int b = lane; b <= len; b += 32) {
    const int64_t j = b == 0 ? i : (int64_t)D.cols[r0 + b - 1];
    const int key = D.perm_dev[j];
    double acc[MD * MD];
    {
      const double *o = bond + R * (r0 + b - 1);
      for (int ss = 0; ss < MD; ss++)
        for (int rr = 0; rr < MD; rr++)
          acc[ss * MD + rr] = b == 0 ? -A[ss * MD + rr] - G[ss] * C[rr]
                                     : o[3 * MD + ss * MD + rr] + G[ss] * o[rr];
    }
    for (int k = 0; k < len; k++) {
      const int64_t kn = D.cols[r0 + k];
      double dth[MD];
      if (kn == j) {
        for (int d = 0; d < MD; d++) dth[d] = 0.;
        for (int64_t q = D.rowptr[kn]; q < D.rowptr[kn + 1]; q++)
          for (int d = 0; d < MD; d++) dth[d] -= bond[R * q + d];
      } else {
        const int p = row_find(D.rowptr, ocols, kn, key);
        if (p < 0) continue;
        for (int d = 0; d < MD; d++) dth[d] = bond[R * (D.rowptr[kn] + p) + d];
      }
      const double *h = bond + R * (r0 + k) + MD;
      for (int ss = 0; ss < MD; ss++)
        for (int rr = 0; rr < MD; rr++) acc[ss * MD + rr] += h[ss] * dth[rr];
    }
    const uint8_t flj = D.flags[j];
    double *blk = J + MD * MD * (r0 + i + b);
    for (int ss = 0; ss < MD; ss++)
      for (int rr = 0; rr < MD; rr++) {
        const bool on = (full || ss == rr) && !dof_fixed(fli, ss, MD) && !dof_fixed(flj, rr, MD);
        blk[ss * MD + rr] = on ? acc[ss * MD + rr] : 0.;
      }
  }
}

// Row node and original column id of every directed bond.
__global__ void k_esqs_topology(int64_t n, const DevPtrs D, int *rows, int *ocols) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int64_t q = D.rowptr[i]; q < D.rowptr[i + 1]; q++) {
    rows[q] = (int)i;
    ocols[q] = D.perm_dev[D.cols[q]];
  }
}

// y = J x over the dofs (identity on fixed ones).
template <int SD>
__global__ void k_esqs_spmv(int64_t n, const DevPtrs D, int mdim, const double *J,
                            const double *x, double *y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  constexpr int S = SD == 2 ? 2 : 4;
  const uint8_t fl = D.flags[i];
  const int64_t r0 = D.rowptr[i];
  const int len = (int)(D.rowptr[i + 1] - r0);
  const int64_t base = r0 + i;
  double acc[3] = {0., 0., 0.};
  for (int b = 0; b <= len; b++) {
    const int64_t j = b == 0 ? i : (int64_t)D.cols[r0 + b - 1];
    const double *blk = J + mdim * mdim * (base + b);
    for (int rr = 0; rr < mdim; rr++) {
      const double xv = x[S * j + rr];
      for (int ss = 0; ss < mdim; ss++) acc[ss] = acc[ss] + blk[mdim * ss + rr] * xv;
    }
  }
  for (int d = 0; d < S; d++) {
    const int64_t q = S * i + d;
    y[q] = (d < 3 && !dof_fixed(fl, d, mdim)) ? acc[d] : x[q];
  }
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
  const unsigned g = blocks_of(P.n, 128);
  if (S == 2) {
    k_esqs_theta<2><<<g, 128, 0, s>>>(P, D, mdim, u, theta);
    k_esqs_force<2><<<g, 128, 0, s>>>(P, D, mdim, u, theta, f);
  } else {
    k_esqs_theta<3><<<g, 128, 0, s>>>(P, D, mdim, u, theta);
    k_esqs_force<3><<<g, 128, 0, s>>>(P, D, mdim, u, theta, f);
  }
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

cudaError_t esqs_topology(const StepParams &P, const DevPtrs &D, int *rows, int *ocols,
                          cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  k_esqs_topology<<<blocks_of(P.n, 128), 128, 0, s>>>(P.n, D, rows, ocols);
  return cudaGetLastError();
}

cudaError_t esqs_jacobian(const StepParams &P, const DevPtrs &D, int S, int mdim, int full,
                          const double *u, const double *theta, double eps, int64_t nnz,
                          const int *rows, const int *ocols, double *bond, double *J,
                          cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  if (nnz > 0) {
    const unsigned g = blocks_of(nnz, 128);
    (S == 2 ? k_esqs_bonds<2> : k_esqs_bonds<3>)<<<g, 128, 0, s>>>(P, D, mdim, rows, nnz, u, theta,
                                                                   eps, bond);
  }
  (mdim == 1   ? k_esqs_rows<1>
   : mdim == 2 ? k_esqs_rows<2>
               : k_esqs_rows<3>)<<<blocks_of(32 * P.n, 128), 128, 0, s>>>(P.n, D, full, ocols,
                                                                          bond, J);
  return cudaGetLastError();
}

cudaError_t esqs_spmv(const StepParams &P, const DevPtrs &D, int S, int mdim, const double *J,
                      const double *x, double *y, cudaStream_t s) {
  if (P.n == 0) return cudaSuccess;
  const unsigned g = blocks_of(P.n, 128);
  if (S == 2)
    k_esqs_spmv<2><<<g, 128, 0, s>>>(P.n, D, mdim, J, x, y);
  else
    k_esqs_spmv<3><<<g, 128, 0, s>>>(P.n, D, mdim, J, x, y);
  return cudaGetLastError();
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
