// qs.cu -- quasi-static Newton solve for RNPBond plates (FP64).
//
// The reference's QuasiStaticModel (src/model/quasistatic/QuasiStaticModel.cpp)
// exists only for ElasticState, with a dense finite-difference Jacobian
// ((N dim)^2 entries, :128-132, :361-454) that does not fit a 40,000-node
// plate.  This solver keeps its load-step / Newton structure (solver :526-594:
// apply loads, residual on free dofs, Newton until the residual norm is below
// tolerance, u += du) with
//   * the residual r = f(u) of FDModel::computeForce (fDModel.cpp:543-582)
//     on free dofs,
//   * the analytic tangent of RNPBond's bond force: for an intact bond with
//     F = k g(S) e, g(S) = S exp(-beta r S^2), S = e.eta / r,
//       dF/du_j = -dF/du_i = A_ij = k g'(S) / r e e^T,
//       g'(S) = (1 - 2 beta r S^2) exp(-beta r S^2),
//     so (-K x)_i = sum_j A_ij (x_i - x_j); 2x2 (or 3x3) symmetric blocks are
//     stored per bond,
//   * block-Jacobi preconditioned conjugate gradients (the reference's
//     default solver tag) on the free dofs, all scalars kept on the device.
// Bonds break as in RNPBond::getBondEF (:263-266): every residual evaluation
// of a Newton iteration marks intact bonds past the critical strain broken and
// leaves them out of that residual.
//
// A load step starts with the displacement-controlled tangent predictor: with
// the tangent K at the previous converged state u and the boundary increment
// du_c, solve K_ff du_f = -(f + K du_c)_f.  (Evaluating f at u + du_c instead
// would put the bonds next to the loaded layer far past the peak of the RNP
// force, where the force, the residual and the stiffness all vanish.)  The
// norm of that right-hand side is the step's residual scale: Newton stops at
// ||f|| <= tol * ||f + K du_c||.  Softening bonds (1 - 2 beta r S^2 < 0)
// are left out of the tangent so the preconditioned CG matrix stays SPD.

#include <algorithm>
#include <functional>
#include <type_traits>
#include <vector>

#include "bond64.cuh"
#include "fd_internal.h"
#include "fp32_common.cuh"
#include "qs_internal.h"
#include "state_io.cuh"

namespace nlm {

// Bond quantities shared by the residual and tangent kernels.
template <int DIM>
__device__ __forceinline__ void qs_bond(const StepParams &P, const double xi[3], const double ui[3],
                                        const double xj[3], const double uj[3], double volj,
                                        double e[3], double &r, double &S, double &k,
                                        double &ex) {
  double dx = xj[0] - xi[0], dy = xj[1] - xi[1], dz = DIM == 3 ? xj[2] - xi[2] : 0.;
  double rr = dx * dx + dy * dy;
  if (DIM == 3) rr = rr + dz * dz;
  r = sqrt(rr);
  double dotp = dx * (uj[0] - ui[0]) + dy * (uj[1] - ui[1]);
  if (DIM == 3) dotp = dotp + dz * (uj[2] - ui[2]);
  S = dotp / rr;
  e[0] = dx / r;
  e[1] = dy / r;
  e[2] = dz / r;
  if (dGT(r, P.check_low)) volj = volj * ((P.check_up - r) / P.h);
  const double infl = influence_d(P, r / P.delta);
  k = infl * 4. * P.C * P.beta / P.invF * volj;
  ex = exp(-P.beta * r * S * S);
}

// Residual (force density on free dofs, zero on fixed dofs); with asm, also
// the tangent blocks of every bond (lower triangle, row-major) and the
// diagonal blocks sum_j A_ij.  Broken bonds contribute nothing.
template <int DIM, bool ASM, bool UPD>
__global__ void k_qs_force(const StepParams P, const DevPtrs D, const double *u, double *res,
                           double *blk, double *dblk, unsigned long long *count) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= P.n) return;
  constexpr int NB = DIM == 2 ? 3 : 6;
  double xi[3], ui[3];
  ld_node<DIM>(D.pos64, i, xi);
  ld_node<DIM>(u, i, ui);
  const uint8_t fl = D.flags[i];
  const int64_t r0 = D.rowptr[i], r1 = D.rowptr[i + 1];
  double fi[3] = {0., 0., 0.};
  double di[6] = {0., 0., 0., 0., 0., 0.};
  int newly = 0;
  for (int64_t q = r0; q < r1; q++) {
    const int kk = (int)(q - r0);
    const int64_t w = (int64_t)(kk >> 5) * P.npad + i;
    const bool fs = (D.bits[w] >> (kk & 31)) & 1u;
    const bool breakable = !(P.nofail && ((fl & FLAG_NOFAIL) || (D.flags[D.cols[q]] & FLAG_NOFAIL)));
    if (fs && breakable) {
      if (ASM)
        for (int c = 0; c < NB; c++) blk[NB * q + c] = 0.;
      continue;
    }
    const int j = D.cols[q];
    double xj[3], uj[3], e[3], r, S, k, ex;
    ld_node<DIM>(D.pos64, j, xj);
    ld_node<DIM>(u, j, uj);
    qs_bond<DIM>(P, xi, ui, xj, uj, D.vol64[j], e, r, S, k, ex);
    if (UPD && breakable && P.irrev && dGT(fabs(S), P.fsc * (P.rbar / sqrt(r)))) {
      D.bits[w] |= 1u << (kk & 31);  // row i is owned by this thread
      newly++;
      if (ASM)
        for (int c = 0; c < NB; c++) blk[NB * q + c] = 0.;
      continue;
    }
    const double s = breakable ? k * S * ex : k * S;
    for (int c = 0; c < DIM; c++) fi[c] += s * e[c];
    if (ASM) {
      const double gp =
          breakable ? k * fmax(1. - 2. * P.beta * r * S * S, 0.) * ex / r : k / r;
      double a[6];
      a[0] = gp * e[0] * e[0];
      a[1] = gp * e[1] * e[0];
      a[2] = gp * e[1] * e[1];
      if (DIM == 3) {
        a[3] = gp * e[2] * e[0];
        a[4] = gp * e[2] * e[1];
        a[5] = gp * e[2] * e[2];
      }
      for (int c = 0; c < NB; c++) {
        blk[NB * q + c] = a[c];
        di[c] += a[c];
      }
    }
  }
  double f[3] = {fi[0], fi[1], fi[2]};
  if (fl & FLAG_FBC) {
    double fe[3];
    ld_node<DIM>(D.fext, i, fe);
    for (int c = 0; c < DIM; c++) f[c] = fe[c] + fi[c];
  }
  for (int c = 0; c < DIM; c++) res[DIM * i + c] = (fl >> c & 1) ? 0. : f[c];
  if (ASM) {
    // relative Levenberg term: keeps blocks of nodes whose remaining bonds
    // are collinear (or gone) invertible
    const double reg = 1e-8 * (DIM == 2 ? 0.5 * (di[0] + di[2]) : (di[0] + di[2] + di[5]) / 3.);
    di[0] += reg;
    di[2] += reg;
    if (DIM == 3) di[5] += reg;
    for (int c = 0; c < NB; c++) dblk[NB * i + c] = di[c];
  }
  if (UPD && newly) atomicAdd(count, (unsigned long long)newly);
}

// The same from the FP64 bond store, G lanes per node: what the reference
// geometry fixes (a square root, four divisions, the volume factor) comes from
// HBM, the FP64 pipe being the bound: 200 x 200 plate, horizon 3h, with tangent:
// k_qs_force took 506 us, 207 FP64 instructions per bond; with this kernel a load
// step (five evaluations) went from 13.7 to 11.9 ms.
template <int DIM, bool ASM, bool UPD, int G>
__global__ void __launch_bounds__(128)
    k_qs_force_bond(const StepParams P, const double kscale, const double nibeta, const DevPtrs D,
                    const double *u, double *res, double *blk, double *dblk,
                    unsigned long long *count) {
  constexpr int NB = DIM == 2 ? 3 : 6;
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  if (i >= P.n) return;
  const int c = threadIdx.x % G;
  const unsigned team = G == 1 ? 0u : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G);
  double ui[3];
  ld_node<DIM>(u, i, ui);
  const int64_t base = D.sell_ptr[i >> 5], r0 = D.rowptr[i];
  const int lane = (int)(i & 31), len = D.rowlen[i];
  const double k0 = P.infl_a0 * 4.;
  double fi[DIM] = {}, di[NB] = {};
  int newly = 0;
  for (int kb = 0; kb < len; kb += 32) {
    uint32_t *wp = D.bits + (int64_t)(kb >> 5) * P.npad + i;
    const uint32_t word = *wp;
    uint32_t cut = 0;
#pragma unroll 2
    for (int k = kb + c; k < min(kb + 32, len); k += G) {
      const int64_t q = base + 32 * (int64_t)k + lane;
      const int j = D.sell_cols[base + 4 * lane + (k >> 2) * 128 + (k & 3)];
      const double2 d = ld_once(D.b64_d + q), e2 = ld_once(D.b64_e + q),
                    rq = ld_once(D.b64_q + q), m = ld_once(D.b64_m + q);
      double2 z = make_double2(0., 0.);
      if (DIM == 3) z = ld_once(D.b64_z + q);
      const int thr = ld_once(D.b64_thr + q);
      const double kk = (D.b64_k ? ld_once(D.b64_k + q) : k0) * kscale * m.y;
      const bool tough = thr < 0;
      double uj[3];
      ld_node<DIM>(u, j, uj);
      double dotp = d.x * (uj[0] - ui[0]) + d.y * (uj[1] - ui[1]);
      if (DIM == 3) dotp = dotp + z.x * (uj[2] - ui[2]);
      const double S = div_by(dotp, rq.x, rq.y);
      bool fs = !tough && ((word >> (k & 31)) & 1u);
      if (UPD && !fs && !tough && P.irrev && hi_abs(S) >= thr &&
          dGT(fabs(S), P.fsc * (P.rbar / sqrt(sqrt(rq.x))))) {
        fs = true;
        cut |= 1u << (k & 31);
        newly++;
      }
      double a[NB] = {};
      if (!fs) {
        const double x = m.x * S * S, ex = tough ? 1. : exp64(x);
        const double e[3] = {e2.x, e2.y, z.y};
        const double s = kk * S * ex;
        for (int h = 0; h < DIM; h++) fi[h] += s * e[h];
        if (ASM) {
          // 1 / r = r / r^2
          double gp = kk * (m.x * nibeta * rq.y);
          if (!tough) gp *= fmax(1. + 2. * x, 0.) * ex;
          int t = 0;
          for (int h = 0; h < DIM; h++)
            for (int g = 0; g <= h; g++, t++) a[t] = gp * e[h] * e[g];
          for (int h = 0; h < NB; h++) di[h] += a[h];
        }
      }
      if (ASM)
        for (int h = 0; h < NB; h++) blk[NB * (r0 + k) + h] = a[h];
    }
    if (UPD) {
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) cut |= __shfl_xor_sync(team, cut, o, G);
      if (cut && c == 0) *wp = word | cut;
    }
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    for (int h = 0; h < DIM; h++) fi[h] += __shfl_xor_sync(team, fi[h], o, G);
    if (ASM)
      for (int h = 0; h < NB; h++) di[h] += __shfl_xor_sync(team, di[h], o, G);
  }
  if (UPD && newly) atomicAdd(count, (unsigned long long)newly);
  if (c) return;
  const uint8_t fl = D.flags[i];
  double fe[3] = {0., 0., 0.};
  if (fl & FLAG_FBC) ld_node<DIM>(D.fext, i, fe);
  for (int h = 0; h < DIM; h++) res[DIM * i + h] = (fl >> h & 1) ? 0. : fe[h] + fi[h];
  if (ASM) {
    // relative Levenberg term, as in k_qs_force
    const double reg = 1e-8 * (DIM == 2 ? 0.5 * (di[0] + di[2]) : (di[0] + di[2] + di[5]) / 3.);
    di[0] += reg;
    di[2] += reg;
    if (DIM == 3) di[5] += reg;
    for (int h = 0; h < NB; h++) dblk[NB * i + h] = di[h];
  }
}

template <typename T>
__device__ __forceinline__ void sym_mul(int dim, const T *a, const T *x, T *y) {
  if (dim == 2) {
    y[0] = a[0] * x[0] + a[1] * x[1];
    y[1] = a[1] * x[0] + a[2] * x[1];
  } else {
    y[0] = a[0] * x[0] + a[1] * x[1] + a[3] * x[2];
    y[1] = a[1] * x[0] + a[2] * x[1] + a[4] * x[2];
    y[2] = a[3] * x[0] + a[4] * x[1] + a[5] * x[2];
  }
}

// Block reduction of one double per thread into part[blockIdx.x].
__device__ __forceinline__ void block_sum(double v, double *part) {
  __shared__ double sh[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = l < (int)(blockDim.x >> 5) ? sh[l] : 0.;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l == 0) part[blockIdx.x] = v;
  }
}

// z = (D_i)^-1 r on the free dofs of node i: the diagonal block b (packed
// symmetric) with the rows and columns of fixed dofs replaced by identity;
// rv is zero on fixed dofs.  A singular block gives z = 0.
template <int DIM, typename T>
__device__ __forceinline__ void block_jacobi(const T *b, uint8_t fl, const T rv[3], T zv[3]) {
  T a[9];
  if (DIM == 2) {
    a[0] = b[0]; a[1] = b[1]; a[2] = b[1]; a[3] = b[2];
  } else {
    a[0] = b[0]; a[1] = b[1]; a[2] = b[3];
    a[3] = b[1]; a[4] = b[2]; a[5] = b[4];
    a[6] = b[3]; a[7] = b[4]; a[8] = b[5];
  }
  for (int c = 0; c < DIM; c++)
    if (fl >> c & 1)
      for (int q = 0; q < DIM; q++) {
        a[c * DIM + q] = (c == q) ? T(1) : T(0);
        a[q * DIM + c] = (c == q) ? T(1) : T(0);
      }
  zv[0] = zv[1] = zv[2] = T(0);
  if (DIM == 2) {
    const T det = a[0] * a[3] - a[1] * a[2];
    if (fabs(det) > T(0)) {
      zv[0] = (a[3] * rv[0] - a[1] * rv[1]) / det;
      zv[1] = (-a[2] * rv[0] + a[0] * rv[1]) / det;
    }
  } else {
    const T c00 = a[4] * a[8] - a[5] * a[7], c01 = a[5] * a[6] - a[3] * a[8],
            c02 = a[3] * a[7] - a[4] * a[6];
    const T det = a[0] * c00 + a[1] * c01 + a[2] * c02;
    if (fabs(det) > T(0)) {
      const T inv[9] = {c00, a[2] * a[7] - a[1] * a[8], a[1] * a[5] - a[2] * a[4],
                             c01, a[0] * a[8] - a[2] * a[6], a[2] * a[3] - a[0] * a[5],
                             c02, a[1] * a[6] - a[0] * a[7], a[0] * a[4] - a[1] * a[3]};
      for (int c = 0; c < 3; c++)
        zv[c] = (inv[3 * c] * rv[0] + inv[3 * c + 1] * rv[1] + inv[3 * c + 2] * rv[2]) / det;
    }
  }
}

// Packed inverse of a node's diagonal block for the FP32 solves, formed in FP64
// (the determinant of a 3-D block, about 1e54 at h = 5e-4 m, is past FP32's
// range); zero rows and columns for fixed dofs.
template <int DIM>
__device__ __forceinline__ void inv_diag32(const double *b, uint8_t fl, float *mi) {
  double inv[3][3];
  for (int c = 0; c < DIM; c++) {
    const double e[3] = {c == 0 ? 1. : 0., c == 1 ? 1. : 0., c == 2 ? 1. : 0.};
    block_jacobi<DIM, double>(b, fl, e, inv[c]);
  }
  int q = 0;
  for (int c = 0; c < DIM; c++)
    for (int d = 0; d <= c; d++, q++)
      mi[q] = (fl >> c & 1) || (fl >> d & 1) ? 0.f : (float)inv[c][d];
}

// Block-Jacobi preconditioner: z_i = (D_i)^-1 r_i on the free dofs of node i
// (fixed dofs removed from the block), plus partial sums of r.z.
template <int DIM>
__global__ void k_qs_precond(const StepParams P, const DevPtrs D, const double *dblk,
                             const double *r, double *z, double *part) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  constexpr int NB = DIM == 2 ? 3 : 6;
  double dot = 0.;
  if (i < P.n) {
    const uint8_t fl = D.flags[i];
    double rv[3] = {0., 0., 0.}, zv[3];
    for (int c = 0; c < DIM; c++) rv[c] = (fl >> c & 1) ? 0. : r[DIM * i + c];
    block_jacobi<DIM, double>(dblk + NB * i, fl, rv, zv);
    for (int c = 0; c < DIM; c++) {
      z[DIM * i + c] = zv[c];
      dot += rv[c] * zv[c];
    }
  }
  block_sum(dot, part);
}

// Sum of partials in a fixed order (deterministic): out = sum part[0..n).
__global__ void k_qs_sum(const double *part, int64_t n, double *out) {
  double v = 0.;
  for (int64_t k = threadIdx.x; k < n; k += blockDim.x) v += part[k];
  __shared__ double sh[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = l < (int)(blockDim.x >> 5) ? sh[l] : 0.;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l == 0) *out = v;
  }
}

// Final stage of a two-stage sum, done by the last block of a launch to
// finish (atomic ticket after a memory fence; no block waits for another).
// The partials are summed in a fixed order (thread t takes t, t + 256, ...,
// then a fixed tree), so the total does not depend on which block is last.
// The ticket counter is reset for the next launch.
__device__ __forceinline__ bool last_block(unsigned *ticket) {
  __shared__ bool is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  return is_last;
}

__device__ __forceinline__ void finish_sums(int nsum, const double *pa, double *ta,
                                            const double *pb, double *tb, unsigned *ticket) {
  __threadfence();
  const int nb = (int)gridDim.x;
  double va = 0., vb = 0.;
  for (int k = threadIdx.x; k < nb; k += blockDim.x) {
    va += __ldcg(pa + k);
    if (nsum > 1) vb += __ldcg(pb + k);
  }
  __shared__ double sh[2][32];
  for (int o = 16; o > 0; o >>= 1) {
    va += __shfl_xor_sync(0xffffffffu, va, o);
    vb += __shfl_xor_sync(0xffffffffu, vb, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sh[0][w] = va;
    sh[1][w] = vb;
  }
  __syncthreads();
  if (w == 0) {
    const bool in = l < (int)(blockDim.x >> 5);
    va = in ? sh[0][l] : 0.;
    vb = in ? sh[1][l] : 0.;
    for (int o = 16; o > 0; o >>= 1) {
      va += __shfl_xor_sync(0xffffffffu, va, o);
      vb += __shfl_xor_sync(0xffffffffu, vb, o);
    }
    if (l == 0) {
      *ta = va;
      if (nsum > 1) *tb = vb;
      *ticket = 0u;
    }
  }
}

// Two block sums at once (partials of block blockIdx.x).
__device__ __forceinline__ void block_sum2(double va, double vb, double *pa, double *pb) {
  __shared__ double sh[2][32];
  for (int o = 16; o > 0; o >>= 1) {
    va += __shfl_xor_sync(0xffffffffu, va, o);
    vb += __shfl_xor_sync(0xffffffffu, vb, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sh[0][w] = va;
    sh[1][w] = vb;
  }
  __syncthreads();
  if (w == 0) {
    const bool in = l < (int)(blockDim.x >> 5);
    va = in ? sh[0][l] : 0.;
    vb = in ? sh[1][l] : 0.;
    for (int o = 16; o > 0; o >>= 1) {
      va += __shfl_xor_sync(0xffffffffu, va, o);
      vb += __shfl_xor_sync(0xffffffffu, vb, o);
    }
    if (l == 0) {
      pa[blockIdx.x] = va;
      pb[blockIdx.x] = vb;
    }
  }
}

// Lanes per node in the tangent products: a row (about 26 bonds at
// horizon 3h) is split over kG lanes so that a 40,000-node plate still puts
// enough warps on every SM to hide the latency of the neighbour gathers.
constexpr int kG = 8;

// One PCG iteration k in two launches.  Vectors: p_k lives in pbuf[k & 1],
// rz_k = r_k.z_k as partials in rzp[k & 1].
// First launch (DIR): beta = rz_k / rz_{k-1}, p_k = z_k + beta p_{k-1} (own
// rows stored, neighbour values formed on the fly from z and p_{k-1}), Ap_k =
// (-K) p_k, partials of p_k.Ap_k.  Without DIR: y = (-K) x with x = z.
template <int DIM, bool DIR>
__global__ void __launch_bounds__(256) k_cg_dir_spmv(
    int64_t n, const uint8_t *flags, const int64_t *rowptr, const int *cols, const double *blk,
    const double *dblk, const double *z, const double *pold, double *pnew, double *ap,
    const double *rz_cur, const double *rz_prev, double *pap_part, unsigned *ticket,
    double *pap_total) {
  double beta = 0.;
  if (DIR) {
    const double rzc = *rz_cur, rzo = *rz_prev;
    beta = rzo != 0. ? rzc / rzo : 0.;
  }
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t i = t / kG;
  const int g = (int)(t % kG);
  constexpr int NB = DIM == 2 ? 3 : 6;
  double acc[3] = {0., 0., 0.}, tv[3];
  if (i < n) {
    const int64_t q1 = rowptr[i + 1];
    for (int64_t q = rowptr[i] + g; q < q1; q += kG) {
      const int j = cols[q];
      double pj[3] = {0., 0., 0.};
      for (int c = 0; c < DIM; c++)
        pj[c] = DIR ? z[DIM * j + c] + beta * pold[DIM * j + c] : z[DIM * j + c];
      sym_mul(DIM, blk + NB * q, pj, tv);
      for (int c = 0; c < DIM; c++) acc[c] -= tv[c];
    }
  }
  for (int o = kG / 2; o > 0; o >>= 1)
    for (int c = 0; c < DIM; c++) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
  double dot = 0.;
  if (i < n && g == 0) {
    const uint8_t fl = flags[i];
    double pi[3] = {0., 0., 0.};
    for (int c = 0; c < DIM; c++) {
      pi[c] = DIR ? z[DIM * i + c] + beta * pold[DIM * i + c] : z[DIM * i + c];
      if (DIR) pnew[DIM * i + c] = pi[c];
    }
    sym_mul(DIM, dblk + NB * i, pi, tv);
    for (int c = 0; c < DIM; c++) {
      const double yc = (fl >> c & 1) ? 0. : acc[c] + tv[c];
      ap[DIM * i + c] = yc;
      dot += pi[c] * yc;
    }
  }
  block_sum(dot, pap_part);
  if (DIR && last_block(ticket)) finish_sums(1, pap_part, pap_total, nullptr, nullptr, ticket);
}

static unsigned grp_blocks(int64_t n) { return (unsigned)((n * kG + 255) / 256); }

int64_t qs_cg_stride(int64_t n) { return (int64_t)grp_blocks(n) + 2; }

// Second launch: alpha = rz_k / p_k.Ap_k, x += alpha p_k, r -= alpha Ap_k,
// z = (D_i)^-1 r (block Jacobi, fixed dofs removed), partials of
// rz_{k+1} = r.z and of r.r.
template <int DIM>
__global__ void k_cg_update(int64_t n, const uint8_t *flags, const double *dblk,
                            const double *p, const double *ap, double *x, double *r, double *z,
                            const double *rz_cur, const double *pap_total, double *rz_part,
                            double *rr_part, unsigned *ticket, double *rz_next,
                            double *rr_total) {
  const double rzc = *rz_cur, pap = *pap_total;
  const double alpha = pap != 0. ? rzc / pap : 0.;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  constexpr int NB = DIM == 2 ? 3 : 6;
  double drz = 0., drr = 0.;
  if (i < n) {
    const uint8_t fl = flags[i];
    double rv[3] = {0., 0., 0.}, zv[3] = {0., 0., 0.};
    for (int c = 0; c < DIM; c++) {
      const int64_t k = DIM * i + c;
      x[k] += alpha * p[k];
      const double rk = r[k] - alpha * ap[k];
      r[k] = rk;
      drr += rk * rk;
      rv[c] = (fl >> c & 1) ? 0. : rk;
    }
    block_jacobi<DIM, double>(dblk + NB * i, fl, rv, zv);
    for (int c = 0; c < DIM; c++) {
      z[DIM * i + c] = zv[c];
      drz += rv[c] * zv[c];
    }
  }
  block_sum2(drz, drr, rz_part, rr_part);
  if (last_block(ticket)) finish_sums(2, rz_part, rz_next, rr_part, rr_total, ticket);
}

__global__ void k_cg_seed(double *rz_prev, double *pold, int64_t m) {
  // rz_{-1} = 1 and p_{-1} = 0 so that p_0 = z_0
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < m) pold[k] = 0.;
  if (k == 0) *rz_prev = 1.;
}

// ---- FP32 Krylov solve ---------------------------------------------------
// The Newton correction only has to cut the residual by lin_tol (1e-4), so
// the tangent blocks, the CG vectors, the SpMV and every per-thread
// operation run in FP32: GB300 issues FP64 at a small fraction of its FP32
// rate, and even a few FP64 operations per thread (a step-length division,
// FP64 partial sums) made these launches FP64-pipe bound.  Block sums are
// formed in FP32 and stored as FP64 partials; the sum over blocks and the
// step lengths alpha, beta are computed in FP64 once per launch, by its last
// block.  The residual, its norm and the Newton update u += dx stay FP64.

__global__ void k_to_f32(int64_t n, const double *a, float *b) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < n) b[k] = (float)a[k];
}
// Tangent blocks to FP32, padded to nb_out floats per bond (16-byte loads).
__global__ void k_blk_to_f32(int64_t nbonds, int nb_in, int nb_out, const double *a, float *b) {
  const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q >= nbonds) return;
  for (int c = 0; c < nb_out; c++) b[nb_out * q + c] = c < nb_in ? (float)a[nb_in * q + c] : 0.f;
}
__global__ void k_to_f64(int64_t n, const float *a, double *b) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < n) b[k] = (double)a[k];
}

__device__ __forceinline__ void block_sum_f(float v, double *part) {
  __shared__ float sh[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = l < (int)(blockDim.x >> 5) ? sh[l] : 0.f;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (l == 0) part[blockIdx.x] = (double)v;
  }
}
__device__ __forceinline__ void block_sum2_f(float va, float vb, double *pa, double *pb) {
  __shared__ float sh[2][32];
  for (int o = 16; o > 0; o >>= 1) {
    va += __shfl_xor_sync(0xffffffffu, va, o);
    vb += __shfl_xor_sync(0xffffffffu, vb, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sh[0][w] = va;
    sh[1][w] = vb;
  }
  __syncthreads();
  if (w == 0) {
    const bool in = l < (int)(blockDim.x >> 5);
    va = in ? sh[0][l] : 0.f;
    vb = in ? sh[1][l] : 0.f;
    for (int o = 16; o > 0; o >>= 1) {
      va += __shfl_xor_sync(0xffffffffu, va, o);
      vb += __shfl_xor_sync(0xffffffffu, vb, o);
    }
    if (l == 0) {
      pa[blockIdx.x] = (double)va;
      pb[blockIdx.x] = (double)vb;
    }
  }
}

template <int DIM>
__global__ void k_inv_diag32(int64_t n, const uint8_t *flags, const double *dblk, float *minv) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  constexpr int NB = DIM == 2 ? 3 : 6;
  if (i < n) inv_diag32<DIM>(dblk + NB * i, flags[i], minv + NB * i);
}

template <int DIM>
__global__ void k_qs_precond32(int64_t n, const float *minv, const float *r, float *z,
                               double *part) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  constexpr int NB = DIM == 2 ? 3 : 6;
  float dot = 0.f;
  if (i < n) {
    float zv[3];
    sym_mul<float>(DIM, minv + NB * i, r + DIM * i, zv);
    for (int c = 0; c < DIM; c++) {
      z[DIM * i + c] = zv[c];
      dot = fmaf(r[DIM * i + c], zv[c], dot);
    }
  }
  block_sum_f(dot, part);
}

// Device scalars of the FP32 CG: tot[0..1] = rz_k by parity, tot[2] = pAp,
// tot[3] = r.r (FP64); fs[0] = alpha, fs[1] = beta (FP32, fs = tot + 4).

// FP32 form of the first CG launch (see k_cg_dir_spmv).  Its last block
// forms alpha_k = rz_k / pAp_k for the second launch.
template <int DIM>
__global__ void __launch_bounds__(256) k_cg32_dir_spmv(
    int64_t n, const uint8_t *flags, const int64_t *rowptr, const int *cols, const float *blk,
    const float *dblk, const float *z, const float *pold, float *pnew, float *ap,
    const double *rz_cur, double *pap_part, unsigned *ticket, double *pap_total, float *fs) {
  const float beta = fs[1];
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t i = t / kG;
  const int g = (int)(t % kG);
  constexpr int NB = DIM == 2 ? 3 : 6;  // diagonal blocks (per node)
  constexpr int NP = DIM == 2 ? 4 : 8;  // bond blocks, padded for 16-byte loads
  float acc[3] = {0.f, 0.f, 0.f}, tv[3];
  if (i < n) {
    const int64_t q1 = rowptr[i + 1];
    // four bonds per pass: all ids, then all gathers, then the products, so
    // that each lane keeps its loads in flight together
    for (int64_t qb = rowptr[i] + g; qb < q1; qb += 4 * kG) {
      int jj[4];
#pragma unroll
      for (int u = 0; u < 4; u++) jj[u] = qb + u * kG < q1 ? cols[qb + u * kG] : -1;
      float bb[4][NP], pj[4][3];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int j = jj[u] < 0 ? (int)i : jj[u];
        const int64_t q = jj[u] < 0 ? qb : qb + u * kG;
        const float4 *bp = reinterpret_cast<const float4 *>(blk + NP * q);
        const float4 b0 = bp[0];
        bb[u][0] = b0.x; bb[u][1] = b0.y; bb[u][2] = b0.z; bb[u][3] = b0.w;
        if (DIM == 3) {
          const float4 b1 = bp[1];
          bb[u][4] = b1.x; bb[u][5] = b1.y; bb[u][6] = b1.z; bb[u][7] = b1.w;
        }
        for (int c = 0; c < DIM; c++) pj[u][c] = fmaf(beta, pold[DIM * j + c], z[DIM * j + c]);
        if (DIM == 2) pj[u][2] = 0.f;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (jj[u] < 0) continue;
        sym_mul<float>(DIM, bb[u], pj[u], tv);
        for (int c = 0; c < DIM; c++) acc[c] -= tv[c];
      }
    }
  }
  for (int o = kG / 2; o > 0; o >>= 1)
    for (int c = 0; c < DIM; c++) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
  float dot = 0.f;
  if (i < n && g == 0) {
    const uint8_t fl = flags[i];
    float pi[3] = {0.f, 0.f, 0.f};
    for (int c = 0; c < DIM; c++) {
      pi[c] = fmaf(beta, pold[DIM * i + c], z[DIM * i + c]);
      pnew[DIM * i + c] = pi[c];
    }
    sym_mul<float>(DIM, dblk + NB * i, pi, tv);
    for (int c = 0; c < DIM; c++) {
      const float yc = (fl >> c & 1) ? 0.f : acc[c] + tv[c];
      ap[DIM * i + c] = yc;
      dot = fmaf(pi[c], yc, dot);
    }
  }
  block_sum_f(dot, pap_part);
  if (last_block(ticket)) {
    finish_sums(1, pap_part, pap_total, nullptr, nullptr, ticket);
    if (threadIdx.x == 0) {
      const double pap = *pap_total;
      fs[0] = (float)(pap != 0. ? *rz_cur / pap : 0.);
    }
  }
}

// FP32 form of the second CG launch (see k_cg_update).  Its last block forms
// beta_k = rz_{k+1} / rz_k for the next first launch.
template <int DIM>
__global__ void k_cg32_update(int64_t n, const float *minv, const float *p,
                              const float *ap, float *x, float *r, float *z,
                              const double *rz_cur, double *rz_part, double *rr_part,
                              unsigned *ticket, double *rz_next, double *rr_total, float *fs) {
  const float alpha = fs[0];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  constexpr int NB = DIM == 2 ? 3 : 6;
  float drz = 0.f, drr = 0.f;
  if (i < n) {
    float rv[3] = {0.f, 0.f, 0.f}, zv[3] = {0.f, 0.f, 0.f};
    for (int c = 0; c < DIM; c++) {
      const int64_t k = DIM * i + c;
      x[k] = fmaf(alpha, p[k], x[k]);
      rv[c] = fmaf(-alpha, ap[k], r[k]);
      r[k] = rv[c];
      drr = fmaf(rv[c], rv[c], drr);
    }
    sym_mul<float>(DIM, minv + NB * i, rv, zv);
    for (int c = 0; c < DIM; c++) {
      z[DIM * i + c] = zv[c];
      drz = fmaf(rv[c], zv[c], drz);
    }
  }
  block_sum2_f(drz, drr, rz_part, rr_part);
  if (last_block(ticket)) {
    finish_sums(2, rz_part, rz_next, rr_part, rr_total, ticket);
    if (threadIdx.x == 0) {
      const double rzc = *rz_cur;
      fs[1] = (float)(rzc != 0. ? *rz_next / rzc : 0.);
    }
  }
}

// ---- the FP32 PCG in one cooperative launch -------------------------------
// At 40,000 nodes the two-launch iteration (27 us: 16.4 + 9.7) is bound by the
// launches, the last-block sums and re-reading the tangent from L2, not by the
// 21 MB it moves.  k_cg32_res runs the whole solve in one launch of one block
// per SM, all resident (cudaLaunchCooperativeKernel), and keeps what a block
// needs on its SM: each block owns a range of consecutive nodes; their tangent
// blocks sit in shared memory with the neighbour's local id (16 bytes per 2-D
// bond, read once per solve), x, r, z and the inverse diagonal block of a node
// in the registers of one thread, and the search direction of the block's
// nodes and of their halo in shared memory, so that an iteration reads nothing
// but the halo's new z.  Halo lists and local ids are laid out once, at
// creation (k_cg_res_setup).
// The two sums of an iteration: a block stores its partial (FP32, as in the
// two-launch form) with the iteration number in one 8-byte word, counts itself
// in, waits for the count and adds all blocks' words in one fixed order, so
// every block forms the same alpha, beta and convergence decision.  A word whose
// number is not yet this iteration's is read again, so only z, which the other
// blocks read after the second sum, needs a fence before the count.  The words
// are added and the step lengths divided in double-float (two-sum) arithmetic:
// an FP64 add takes 67 cycles here, a division 566, and they sit on the one
// chain everything waits for.  (152 SMs polling each other's words instead of
// one counter took 7,500 cycles per sum, with one array or with a private
// mailbox per block alike; the counter and the read 3,400.)
// A poll is bounded (wait_ns of globaltimer); one that runs out sets status =
// NLM_ERR_TIMEOUT and every block leaves at its next poll, so the launch
// always ends.
// Range: the words and their double-float sums end at 3.4e38, where the
// two-launch form's totals (FP64) go on.  A right-hand side whose r.r leaves
// 2^-60 .. 2^90 is scaled by a power of two to r.r near 2^40 or 2^88 (no further
// from above: r.z is r.r over the stiffness, which is large then), the same bits as
// without wherever those stay in range (r.r of the plate below is 1e21 in N and m).
// Bound of the step lengths: over 4,000 random sets of 152 and 1,256 words the FP32
// quotient of the double-float sums equals that of FP64 sums in all of them.
// 200 x 200 plate, horizon 3h: 7 us per iteration, of which the
// two sums take 4 (counting in, the skew of the blocks, reading the words), the
// product 1.4 and the halo 0.8; a load step 38.0 -> 13.7 ms.

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr int kResThreads = 1024;
constexpr int kResHash = 2 * kResHalo;

// Halo list (ids of the nodes outside the block's range that its rows meet)
// and, per bond, the local id of its neighbour: own nodes first, then the
// halo.  nh < 0: more than kResHalo of them.
__global__ void __launch_bounds__(kResThreads)
    k_cg_res_setup(int64_t n, int nb, const int64_t *rowptr, const int *cols, int *halo, int *nh,
                   uint16_t *lid) {
  __shared__ int keys[kResHash], vals[kResHash], count;
  const int64_t n0 = (int64_t)blockIdx.x * nb, n1 = min(n0 + nb, n);
  for (int k = threadIdx.x; k < kResHash; k += kResThreads) keys[k] = -1;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  auto slot_of = [&](int j) { return (int)(((unsigned)j * 2654435761u) >> 16) % kResHash; };
  const int64_t q0 = rowptr[n0], q1 = rowptr[n1];
  for (int64_t q = q0 + threadIdx.x; q < q1; q += kResThreads) {
    const int j = cols[q];
    if (j >= n0 && j < n1) continue;
    int s = slot_of(j);
    for (int t = 0; t < kResHash; t++, s = (s + 1) % kResHash) {
      const int old = atomicCAS(keys + s, -1, j);
      if (old == j) break;
      if (old == -1) {
        const int k = atomicAdd(&count, 1);
        vals[s] = k;
        if (k < kResHalo) halo[blockIdx.x * kResHalo + k] = j;
        break;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) nh[blockIdx.x] = count <= kResHalo ? count : -1;
  if (count > kResHalo) return;
  for (int64_t q = q0 + threadIdx.x; q < q1; q += kResThreads) {
    const int j = cols[q];
    int id = (int)(j - n0);
    if (j < n0 || j >= n1) {
      int s = slot_of(j);
      while (keys[s] != j) s = (s + 1) % kResHash;  // present
      id = nb + vals[s];
    }
    lid[q] = (uint16_t)id;
  }
}

// Scale of a right-hand side with this r.r, as an exponent (see above); 0 for an
// r.r of zero, infinity or NaN.
__device__ __forceinline__ int res_exponent(double rr0) {
  const int hi = __double2hiint(rr0), e = (hi >> 20) - 1023;
  if (hi <= 0 || e == 1024 || (e >= -60 && e < 90)) return 0;
  return ((e > 0 ? 88 : 40) - max(e, -1022)) >> 1;
}
__device__ __forceinline__ double exp2i(int e) {  // |e| <= 1022
  return __hiloint2double((e + 1023) << 20, 0);
}

// Warp 0: publish N partials, wait for all blocks, sum their words in one fixed
// order; false when a wait ran out or another block gave up.  fence: what the
// block wrote before is visible to a block that has returned.
template <int N, bool FENCE>
__device__ __forceinline__ bool res_sum(const CgRes &A, int slot, uint32_t epoch, uint32_t arrivals,
                                        const float v[N], df sum[N]) {
  const int lane = threadIdx.x;
  bool ok = true;
  if (lane == 0) {
    if (FENCE) __threadfence();
    for (int a = 0; a < N; a++)
      *(volatile unsigned long long *)(A.words + (slot + a) * A.stride + blockIdx.x) =
          ((unsigned long long)epoch << 32) | __float_as_uint(v[a]);
    atomicAdd(A.count, 1u);
  }
  uint64_t t0 = 0;
  int polls = 0;
  // the time and the other blocks' status every 64 polls
  auto give_up = [&]() {
    if ((++polls & 63) == 0) {
      if (*(volatile const int *)A.status != 0) return true;
      const uint64_t now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > A.wait_ns) {
        atomicExch(A.status, NLM_ERR_TIMEOUT);
        return true;
      }
    }
    return false;
  };
  if (lane == 0)
    while (ok && *(volatile const unsigned *)A.count < arrivals) ok = !give_up();
  ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
  if (FENCE) __threadfence();
  for (int a = 0; a < N; a++) sum[a] = df{0.f, 0.f};
  for (int b0 = lane; b0 < A.blocks; b0 += 160) {
    unsigned long long w[5][N];
    bool all = true;
    do {
      all = true;
#pragma unroll
      for (int u = 0; u < 5; u++)
#pragma unroll
        for (int a = 0; a < N; a++) {
          const int b = min(b0 + 32 * u, A.blocks - 1);
          w[u][a] = *(volatile const unsigned long long *)(A.words + (slot + a) * A.stride + b);
          all = all && (uint32_t)(w[u][a] >> 32) == epoch;
        }
      if (!all && ok) ok = !give_up();
    } while (!all && ok);
#pragma unroll
    for (int u = 0; u < 5; u++)
#pragma unroll
      for (int a = 0; a < N; a++)
        if (b0 + 32 * u < A.blocks)
          sum[a] = df_add(sum[a], df{__uint_as_float((uint32_t)w[u][a]), 0.f});
  }
  ok = __all_sync(0xffffffffu, ok);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < N; a++) {
      const df q{__shfl_xor_sync(0xffffffffu, sum[a].hi, o),
                 __shfl_xor_sync(0xffffffffu, sum[a].lo, o)};
      sum[a] = df_add(sum[a], q);
    }
  return ok;
}

// a / b rounded to FP32 (a quotient of the leading parts and its correction).
__device__ __forceinline__ float df_div(df a, df b) {
  const float q = __fdiv_rn(a.hi, b.hi);
  const float r = fmaf(-q, b.hi, a.hi) + fmaf(-q, b.lo, a.lo);
  const float c = __fdiv_rn(r, b.hi);
  return isfinite(c) ? q + c : q;
}

// Block sums of N floats; warp 0's lanes end with them.  Ends with warp 0
// alone past a block barrier.
template <int N>
__device__ __forceinline__ void res_block_sum(float v[N], float (*sh)[32]) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < N; a++) v[a] += __shfl_xor_sync(0xffffffffu, v[a], o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0)
    for (int a = 0; a < N; a++) sh[a][w] = v[a];
  __syncthreads();
  if (w == 0) {
    for (int a = 0; a < N; a++) v[a] = sh[a][l];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int a = 0; a < N; a++) v[a] += __shfl_xor_sync(0xffffffffu, v[a], o);
  }
}

// res[0] = iterations done, res[1] = 1 where r.r reached its target (0 where it
// became a NaN or an infinity)
template <int DIM>
__global__ void __launch_bounds__(kResThreads, 1) k_cg32_res(const CgRes A) {
  constexpr int NB = DIM == 2 ? 3 : 6;
  constexpr int NW = DIM == 2 ? 1 : 2;  // float4 words per bond
  extern __shared__ float4 s_bond[];
  __shared__ float s_red[2][32];
  __shared__ float s_scal;
  __shared__ int s_stop;
  const int64_t n0 = (int64_t)blockIdx.x * A.nb;
  const int own = (int)(min(n0 + A.nb, A.n) - n0);
  // lanes in turn: the m-th bond of a lane is word (warp * M + m) * 32 + lane, so
  // that a warp's reads are consecutive
  float *s_p = reinterpret_cast<float *>(s_bond + (size_t)NW * 32 * A.warps * A.bonds_per_lane);
  const int nh = A.nh[blockIdx.x];
  const int *halo = A.halo + (int64_t)blockIdx.x * kResHalo;
  for (int k = threadIdx.x; k < DIM * (A.nb + nh); k += kResThreads) s_p[k] = 0.f;
  // L lanes per node, the first of them its owner
  const int L = A.lanes, tpw = 32 / L, lane = threadIdx.x & 31;
  const int t = (threadIdx.x >> 5) * tpw + lane / L, l = lane % L;
  const bool team = lane < tpw * L && t < own;
  const bool lead = team && l == 0;
  const int64_t i = n0 + t;
  const double rscale = exp2i(res_exponent(*A.rr0));
  float x[DIM] = {}, r[DIM] = {}, z[DIM] = {}, dg[NB] = {}, mi[NB] = {};
  bool fixed[DIM] = {};
  int nk = 0;
  float4 *bonds = s_bond + NW * ((size_t)(threadIdx.x >> 5) * A.bonds_per_lane * 32 + lane);
  if (team) {
    const int64_t r0 = A.rowptr[i] + l, r1 = A.rowptr[i + 1];
    for (int64_t q = r0; q < r1; q += L, nk++) {
      const double *b = A.blk + NB * q;
      const float id = __int_as_float(A.lid[q]);
      bonds[NW * 32 * nk] = make_float4((float)b[0], (float)b[1], (float)b[2],
                                        DIM == 2 ? id : (float)b[3]);
      if (DIM == 3) bonds[NW * 32 * nk + 1] = make_float4((float)b[4], (float)b[5], id, 0.f);
    }
  }
  if (lead) {
    const uint8_t fl = A.flags[i];
    double b[NB];
    for (int c = 0; c < NB; c++) {
      b[c] = A.dblk[NB * i + c];
      dg[c] = (float)b[c];
    }
    inv_diag32<DIM>(b, fl, mi);
    for (int c = 0; c < DIM; c++) {
      fixed[c] = fl >> c & 1;
      r[c] = (float)(A.rhs[DIM * i + c] * rscale);
    }
  }
  // The target in FP32, two steps below tol^2 r.r at most, so that a sum rounded to
  // FP32 is not above it only where the sum itself is not; no limit where there is
  // nothing to do.
  const double rr1 = *A.rr0 * rscale * rscale, goal = A.tol2 * rr1;
  const float below = __double2float_rd(goal);
  const float target = !(rr1 > goal) ? INFINITY
                       : below > 0.f ? __uint_as_float(__float_as_uint(below) - 1u)
                                     : 0.f;
  float rr = (float)rr1;
  df rz{0.f, 0.f};
  float beta = 0.f;
  int it = 0;
  uint32_t epoch = A.epoch + 1, arrivals = 0;
  const uint32_t all = (uint32_t)(A.blocks + A.extra);
  if (threadIdx.x == 0) s_stop = 0;
  // z = M^-1 r, published with r.z and r.r; beta and the decision to go on
  auto precondition = [&]() {
    float v[2] = {0.f, 0.f};
    if (lead) {
      sym_mul<float>(DIM, mi, r, z);
      for (int c = 0; c < DIM; c++) {
        A.z[DIM * i + c] = z[c];
        v[0] = fmaf(r[c], z[c], v[0]);
        v[1] = fmaf(r[c], r[c], v[1]);
      }
    }
    res_block_sum<2>(v, s_red);
    if (threadIdx.x < 32) {
      df s[2];
      const bool ok = res_sum<2, true>(A, 1, epoch, arrivals += all, v, s);
      if (it > 0) rr = s[1].hi;
      if (threadIdx.x == 0) {
        s_scal = it > 0 && rz.hi != 0.f ? df_div(s[0], rz) : 0.f;
        s_stop = !ok ? 2 : !(rr > target) || it >= A.max_iters ? 1 : 0;
      }
      rz = s[0];
    }
    __syncthreads();
    beta = s_scal;
  };
  precondition();
  while (s_stop == 0) {
    epoch++;
    float p[DIM];
    if (lead)
      for (int c = 0; c < DIM; c++)
        s_p[DIM * t + c] = p[c] = fmaf(beta, s_p[DIM * t + c], z[c]);
    for (int h = threadIdx.x; h < nh; h += kResThreads) {
      const int64_t g = halo[h];
      float *ph = s_p + DIM * (A.nb + h);
      if (DIM == 2) {
        const float2 zz = __ldcg(reinterpret_cast<const float2 *>(A.z) + g);
        ph[0] = fmaf(beta, ph[0], zz.x);
        ph[1] = fmaf(beta, ph[1], zz.y);
      } else {
        for (int c = 0; c < DIM; c++) ph[c] = fmaf(beta, ph[c], __ldcg(A.z + DIM * g + c));
      }
    }
    __syncthreads();
    float acc[DIM] = {}, tv[DIM], ap[DIM] = {};
#pragma unroll 2
    for (int k = 0; k < nk; k++) {
      const float4 w = bonds[NW * 32 * k];
      if (DIM == 2) {
        const float2 pj = reinterpret_cast<const float2 *>(s_p)[__float_as_int(w.w)];
        acc[0] -= fmaf(w.x, pj.x, w.y * pj.y);
        acc[1] -= fmaf(w.y, pj.x, w.z * pj.y);
      } else {
        const float4 w1 = bonds[NW * 32 * k + 1];
        const float a[6] = {w.x, w.y, w.z, w.w, w1.x, w1.y};
        sym_mul<float>(DIM, a, s_p + DIM * __float_as_int(w1.z), tv);
        for (int c = 0; c < DIM; c++) acc[c] -= tv[c];
      }
    }
    for (int c = 0; c < DIM; c++) {
      const float mine = acc[c];
      for (int o = 1; o < L; o++) acc[c] += __shfl_down_sync(0xffffffffu, mine, o);
    }
    float dot[1] = {0.f};
    if (lead) {
      sym_mul<float>(DIM, dg, p, tv);
      for (int c = 0; c < DIM; c++) {
        ap[c] = fixed[c] ? 0.f : acc[c] + tv[c];
        dot[0] = fmaf(p[c], ap[c], dot[0]);
      }
    }
    res_block_sum<1>(dot, s_red);
    if (threadIdx.x < 32) {
      df s[1];
      const bool ok = res_sum<1, false>(A, 0, epoch, arrivals += all, dot, s);
      if (threadIdx.x == 0) {
        s_scal = s[0].hi != 0.f ? df_div(rz, s[0]) : 0.f;
        if (!ok) s_stop = 2;
      }
    }
    __syncthreads();
    if (s_stop) break;
    const float alpha = s_scal;
    it++;
    if (lead)
      for (int c = 0; c < DIM; c++) {
        x[c] = fmaf(alpha, p[c], x[c]);
        r[c] = fmaf(-alpha, ap[c], r[c]);
      }
    precondition();
  }
  if (lead) {
    const double back = exp2i(-res_exponent(*A.rr0));
    for (int c = 0; c < DIM; c++) A.dx[DIM * i + c] = (double)x[c] * back;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    A.res[0] = (double)it;
    A.res[1] = rr <= target && isfinite(rr) ? 1. : 0.;
  }
}

__global__ void k_cg32_seed(float *fs, float *pold, int64_t m) {
  // beta = 0 for the first direction (p_0 = z_0); p_{-1} = 0
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < m) pold[k] = 0.f;
  if (k == 0) fs[1] = 0.f;
}

// u_full (S doubles per node) <-> dof vectors (DIM per node).
template <int DIM>
__global__ void k_qs_add(int64_t n, const double *du, double *u) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int c = 0; c < DIM; c++) u[(DIM == 2 ? 2 : 4) * i + c] += du[DIM * i + c];
}

static unsigned qblk(int64_t n) { return (unsigned)((n + 255) / 256); }

template <int DIM>
static void qs_force_dim(const StepParams &P, const DevPtrs &D, const double *u, double *res,
                         double *blk, double *dblk, bool assemble, unsigned long long *count,
                         cudaStream_t s) {
  if (D.b64_d) {
    // four lanes per node until one thread per node fills the chip: us per load
    // step of three evaluations with one / four lanes, 2-D horizon 3h -- 400 nodes
    // 442 / 331, 10,000: 475 / 428, 40,000: 774 / 696, 90,000: 1149 / 1110, 129,600:
    // 1445 / 1430, 250,000: 2426 / 2466, 490,000: 4436 / 4442
    const int G = P.n < 131072 ? 4 : 1;
    const unsigned g = (unsigned)((P.n * G + 127) / 128);
    const double ks = P.C * P.beta / P.invF, nib = -1. / P.beta;
    auto go = [&](auto a, auto c, auto team) {
      k_qs_force_bond<DIM, decltype(a)::value, decltype(c)::value, decltype(team)::value>
          <<<g, 128, 0, s>>>(P, ks, nib, D, u, res, blk, dblk, count);
    };
    auto pick = [&](auto a, auto c) {
      if (G == 4)
        go(a, c, std::integral_constant<int, 4>{});
      else
        go(a, c, std::integral_constant<int, 1>{});
    };
    const std::true_type y{};
    const std::false_type no{};
    if (assemble)
      count ? pick(y, y) : pick(y, no);
    else
      count ? pick(no, y) : pick(no, no);
    return;
  }
  if (assemble && count)
    k_qs_force<DIM, true, true><<<qblk(P.n), 256, 0, s>>>(P, D, u, res, blk, dblk, count);
  else if (assemble)
    k_qs_force<DIM, true, false><<<qblk(P.n), 256, 0, s>>>(P, D, u, res, blk, dblk, count);
  else if (count)
    k_qs_force<DIM, false, true><<<qblk(P.n), 256, 0, s>>>(P, D, u, res, blk, dblk, count);
  else
    k_qs_force<DIM, false, false><<<qblk(P.n), 256, 0, s>>>(P, D, u, res, blk, dblk, count);
}

cudaError_t qs_residual(const StepParams &P, const DevPtrs &D, const double *u, double *res,
                        double *blk, double *dblk, bool assemble, cudaStream_t s,
                        unsigned long long *count) {
  if (P.n == 0) return cudaSuccess;
  if (P.dim == 2)
    qs_force_dim<2>(P, D, u, res, blk, dblk, assemble, count, s);
  else
    qs_force_dim<3>(P, D, u, res, blk, dblk, assemble, count, s);
  return cudaGetLastError();
}

cudaError_t qs_dot(const double *a, const double *b, int64_t m, double *part, double *out,
                   cudaStream_t s);

__global__ void k_qs_dot(int64_t m, const double *a, const double *b, double *part) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  block_sum(k < m ? a[k] * b[k] : 0., part);
}

cudaError_t qs_dot(const double *a, const double *b, int64_t m, double *part, double *out,
                   cudaStream_t s) {
  const unsigned g = qblk(m);
  k_qs_dot<<<g, 256, 0, s>>>(m, a, b, part);
  k_qs_sum<<<1, 256, 0, s>>>(part, g, out);
  return cudaGetLastError();
}

// Preconditioned CG on (-K) dx = r (free dofs).  Scalars: sc[0] = rz_old,
// sc[1] = pAp, sc[2] = rz_new, sc[3] = r.r (convergence check).
static cudaError_t qs_cg64(const StepParams &P, const DevPtrs &D, const QSWork &W, const double *rhs,
                  double *dx, double tol, int max_iters, int check_every, int *iters,
                  cudaStream_t s) {
  const int dim = P.dim;
  const int64_t m = (int64_t)dim * P.n;
  const unsigned gn = qblk(P.n), gg = grp_blocks(P.n);
  const int64_t stride = qs_cg_stride(P.n);
  // partials: pAp (K1 blocks), rz and r.r (K2 blocks); totals on the device:
  // rz_k in tot[k & 1], pAp in tot[2], r.r in tot[3]
  double *pap_p = W.cgpart, *rz_p = W.cgpart + stride, *rr_p = W.cgpart + 2 * stride;
  double *tot = W.cgs;
  double *pbuf[2] = {W.p, W.p2};
  cudaError_t e;
  if ((e = cudaMemsetAsync(dx, 0, sizeof(double) * m, s))) return e;
  if ((e = cudaMemcpyAsync(W.r, rhs, sizeof(double) * m, cudaMemcpyDeviceToDevice, s))) return e;
  // z_0 = M^-1 r_0 and rz_0; rz_{-1} = 1, p_{-1} = 0
  if (dim == 2)
    k_qs_precond<2><<<gn, 256, 0, s>>>(P, D, W.dblk, W.r, W.z, rz_p);
  else
    k_qs_precond<3><<<gn, 256, 0, s>>>(P, D, W.dblk, W.r, W.z, rz_p);
  k_qs_sum<<<1, 256, 0, s>>>(rz_p, gn, tot + 0);
  k_cg_seed<<<qblk(m), 256, 0, s>>>(tot + 1, pbuf[1], m);
  double rr0 = 0.;
  if ((e = qs_dot(W.r, W.r, m, W.part, W.sc + 3, s))) return e;
  if ((e = cudaMemcpyAsync(&rr0, W.sc + 3, sizeof(double), cudaMemcpyDeviceToHost, s))) return e;
  if ((e = cudaStreamSynchronize(s))) return e;
  const double target = tol * tol * rr0;
  int it = 0;
  if (rr0 == 0.) {
    *iters = 0;
    return cudaSuccess;
  }
  while (it < max_iters) {
    for (int q = 0; q < check_every && it < max_iters; q++, it++) {
      const int cur = it & 1, prv = cur ^ 1;
      if (dim == 2) {
        k_cg_dir_spmv<2, true><<<gg, 256, 0, s>>>(P.n, D.flags, D.rowptr, D.cols, W.blk,
                                                  W.dblk, W.z, pbuf[prv], pbuf[cur], W.ap,
                                                  tot + cur, tot + prv, pap_p, W.ticket,
                                                  tot + 2);
        k_cg_update<2><<<gn, 256, 0, s>>>(P.n, D.flags, W.dblk, pbuf[cur], W.ap, dx, W.r, W.z,
                                          tot + cur, tot + 2, rz_p, rr_p, W.ticket + 1,
                                          tot + prv, tot + 3);
      } else {
        k_cg_dir_spmv<3, true><<<gg, 256, 0, s>>>(P.n, D.flags, D.rowptr, D.cols, W.blk,
                                                  W.dblk, W.z, pbuf[prv], pbuf[cur], W.ap,
                                                  tot + cur, tot + prv, pap_p, W.ticket,
                                                  tot + 2);
        k_cg_update<3><<<gn, 256, 0, s>>>(P.n, D.flags, W.dblk, pbuf[cur], W.ap, dx, W.r, W.z,
                                          tot + cur, tot + 2, rz_p, rr_p, W.ticket + 1,
                                          tot + prv, tot + 3);
      }
    }
    if ((e = cudaGetLastError())) return e;
    double rr = 0.;
    if ((e = cudaMemcpyAsync(&rr, tot + 3, sizeof(double), cudaMemcpyDeviceToHost, s))) return e;
    if ((e = cudaStreamSynchronize(s))) return e;
    if (!(rr > target)) break;
  }
  *iters = it;
  return cudaGetLastError();
}

static cudaError_t qs_cg32(const StepParams &P, const DevPtrs &D, const QSWork &W,
                           const double *rhs, double *dx, double tol, int max_iters,
                           int check_every, int *iters, bool *converged, cudaStream_t s) {
  *converged = false;
  const int dim = P.dim;
  const int64_t m = (int64_t)dim * P.n;
  const unsigned gn = qblk(P.n), gg = grp_blocks(P.n);
  const int64_t stride = qs_cg_stride(P.n);
  // partials: pAp (K1 blocks), rz and r.r (K2 blocks); totals on the device:
  // rz_k in tot[k & 1], pAp in tot[2], r.r in tot[3]
  double *pap_p = W.cgpart, *rz_p = W.cgpart + stride, *rr_p = W.cgpart + 2 * stride;
  double *tot = W.cgs;
  float *fs = reinterpret_cast<float *>(tot + 4);
  float *pbuf[2] = {W.p32, W.p32b};
  const int NB = dim == 2 ? 3 : 6;
  cudaError_t e;
  // FP32 copies of the tangent and of the right-hand side; x = 0
  k_blk_to_f32<<<qblk(W.nnz + 1), 256, 0, s>>>(W.nnz + 1, NB, dim == 2 ? 4 : 8, W.blk, W.blk32);
  k_to_f32<<<qblk((int64_t)NB * P.n), 256, 0, s>>>((int64_t)NB * P.n, W.dblk, W.dblk32);
  k_to_f32<<<qblk(m), 256, 0, s>>>(m, rhs, W.r32);
  if ((e = cudaMemsetAsync(W.x32, 0, sizeof(float) * m, s))) return e;
  // z_0 = M^-1 r_0 and rz_0; beta_{-1} = 0, p_{-1} = 0
  if (dim == 2) {
    k_inv_diag32<2><<<gn, 256, 0, s>>>(P.n, D.flags, W.dblk, W.minv32);
    k_qs_precond32<2><<<gn, 256, 0, s>>>(P.n, W.minv32, W.r32, W.z32, rz_p);
  } else {
    k_inv_diag32<3><<<gn, 256, 0, s>>>(P.n, D.flags, W.dblk, W.minv32);
    k_qs_precond32<3><<<gn, 256, 0, s>>>(P.n, W.minv32, W.r32, W.z32, rz_p);
  }
  k_qs_sum<<<1, 256, 0, s>>>(rz_p, gn, tot + 0);
  k_cg32_seed<<<qblk(m), 256, 0, s>>>(fs, pbuf[1], m);
  double rr0 = 0.;
  if ((e = qs_dot(rhs, rhs, m, W.part, W.sc + 3, s))) return e;
  if ((e = cudaMemcpyAsync(&rr0, W.sc + 3, sizeof(double), cudaMemcpyDeviceToHost, s))) return e;
  if ((e = cudaStreamSynchronize(s))) return e;
  const double target = tol * tol * rr0;
  int it = 0;
  if (rr0 == 0.) {
    *iters = 0;
    *converged = true;
    return cudaMemsetAsync(dx, 0, sizeof(double) * m, s);
  }
  while (it < max_iters) {
    for (int q = 0; q < check_every && it < max_iters; q++, it++) {
      const int cur = it & 1, prv = cur ^ 1;
      if (dim == 2) {
        k_cg32_dir_spmv<2><<<gg, 256, 0, s>>>(P.n, D.flags, D.rowptr, D.cols, W.blk32,
                                              W.dblk32, W.z32, pbuf[prv], pbuf[cur], W.ap32,
                                              tot + cur, pap_p, W.ticket, tot + 2, fs);
        k_cg32_update<2><<<gn, 256, 0, s>>>(P.n, W.minv32, pbuf[cur], W.ap32, W.x32,
                                            W.r32, W.z32, tot + cur, rz_p, rr_p, W.ticket + 1,
                                            tot + prv, tot + 3, fs);
      } else {
        k_cg32_dir_spmv<3><<<gg, 256, 0, s>>>(P.n, D.flags, D.rowptr, D.cols, W.blk32,
                                              W.dblk32, W.z32, pbuf[prv], pbuf[cur], W.ap32,
                                              tot + cur, pap_p, W.ticket, tot + 2, fs);
        k_cg32_update<3><<<gn, 256, 0, s>>>(P.n, W.minv32, pbuf[cur], W.ap32, W.x32,
                                            W.r32, W.z32, tot + cur, rz_p, rr_p, W.ticket + 1,
                                            tot + prv, tot + 3, fs);
      }
    }
    if ((e = cudaGetLastError())) return e;
    double rr = 0.;
    if ((e = cudaMemcpyAsync(&rr, tot + 3, sizeof(double), cudaMemcpyDeviceToHost, s))) return e;
    if ((e = cudaStreamSynchronize(s))) return e;
    if (!(rr > target)) {
      *converged = rr <= target;  // not where r.r became a NaN
      break;
    }
  }
  k_to_f64<<<qblk(m), 256, 0, s>>>(m, W.x32, dx);
  *iters = it;
  return cudaGetLastError();
}

// The whole FP32 solve in one cooperative launch; *status = NLM_ERR_TIMEOUT
// when a wait ran out (dx is then undefined).
static cudaError_t qs_cg32_res(const StepParams &P, const DevPtrs &D, QSWork &W,
                               const double *rhs, double *dx, double tol, int max_iters,
                               int *iters, bool *converged, int *status, cudaStream_t s) {
  cudaError_t e = qs_dot(rhs, rhs, (int64_t)P.dim * P.n, W.part, W.sc + 3, s);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(W.kr.status, 0, 2 * sizeof(int), s);  // and the count
  if (e != cudaSuccess) return e;
  // iteration numbers go on from solve to solve, so no word holds one that a
  // later solve waits for
  if (W.epoch > 0xffffffffu - (uint32_t)max_iters - 4) {
    e = cudaMemsetAsync(W.kr.words, 0, sizeof(uint64_t) * 3 * W.kr.stride, s);
    if (e != cudaSuccess) return e;
    W.epoch = 0;
  }
  CgRes A = W.kr;
  A.epoch = W.epoch;
  W.epoch += (uint32_t)max_iters + 2;
  A.rhs = rhs;
  A.dx = dx;
  A.rr0 = W.sc + 3;
  A.tol2 = tol * tol;
  A.max_iters = max_iters;
  void *args[] = {&A};
  e = cudaLaunchCooperativeKernel(
      P.dim == 2 ? (const void *)k_cg32_res<2> : (const void *)k_cg32_res<3>, A.blocks,
      kResThreads, args, W.res_smem, s);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
    // fewer SMs to be had than at creation: the two-launch form
    cudaGetLastError();
    W.kr.blocks = 0;
    return cudaSuccess;
  }
  double r[2] = {};
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(r, A.res, sizeof(r), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(status, A.status, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess || *status != 0) return e;
  *iters = (int)r[0];
  *converged = r[1] != 0.;
  return cudaSuccess;
}

// Layout of the resident solve: blocks, node ranges, lanes per node, halo
// lists.  blocks = 0 where it does not apply: no cooperative launch, or a
// block's tangent (16 bytes per 2-D bond, 32 per 3-D one) or halo that does
// not fit its SM -- above about 1.8 million 2-D bonds the tangent streams from
// L2 in the two-launch form.
cudaError_t qs_res_setup(const StepParams &P, const DevPtrs &D, const int64_t *rowptr_host,
                         QSWork &W, const std::function<cudaError_t(void **, size_t)> &alloc,
                         cudaStream_t s) {
  CgRes &A = W.kr;
  A.blocks = 0;
  int dev = 0, sms = 0, coop = 0, smem = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (!coop || sms <= 0 || P.n == 0) return cudaSuccess;
  const int64_t n = P.n;
  int64_t longest = 0;
  for (int64_t k = 0; k < n; k++)
    longest = std::max(longest, rowptr_host[k + 1] - rowptr_host[k]);
  // at least 64 nodes per block (fewer words to add), unless their tangent
  // does not fit
  int nb = 0, blocks = 0, L = 0, warps = 0, M = 0;
  size_t words = 0;
  smem -= 1024;  // the kernel's static arrays
  for (int64_t most : {(n + 63) / 64, n}) {
    const int64_t want = std::min<int64_t>(sms, most);
    nb = (int)std::min<int64_t>((n + want - 1) / want, 1 << 20);
    blocks = (int)((n + nb - 1) / nb);
    L = 8;
    while (L > 1 && 32 / L * (kResThreads / 32) < nb) L--;
    warps = (nb + 32 / L - 1) / (32 / L);
    M = (int)((longest + L - 1) / L);
    words = (size_t)(P.dim == 2 ? 16 : 32) * 32 * warps * M;
    if (nb <= kResThreads && words <= (size_t)smem) break;
  }
  if (nb > kResThreads || words > (size_t)smem) return cudaSuccess;
  const int64_t nnz = rowptr_host[n];
  void *p[6] = {};
  const size_t bytes[6] = {sizeof(int) * (size_t)blocks * kResHalo, sizeof(int) * (size_t)blocks,
                           sizeof(uint16_t) * (size_t)(nnz + 1),
                           sizeof(uint64_t) * (3 * (size_t)blocks + 1),
                           sizeof(float) * (size_t)P.dim * n, sizeof(double) * 4};
  for (int k = 0; k < 6; k++)
    if ((e = alloc(&p[k], bytes[k])) != cudaSuccess) return e;
  std::vector<int> nh(blocks);
  k_cg_res_setup<<<blocks, kResThreads, 0, s>>>(n, nb, D.rowptr, D.cols, (int *)p[0], (int *)p[1],
                                                (uint16_t *)p[2]);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(nh.data(), p[1], bytes[1], cudaMemcpyDeviceToHost, s))) return e;
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
  int hmax = 0;
  for (int v : nh) {
    if (v < 0) return cudaSuccess;
    hmax = std::max(hmax, v);
  }
  W.res_smem = words + sizeof(float) * P.dim * (size_t)(nb + hmax);
  const void *kern = P.dim == 2 ? (const void *)k_cg32_res<2> : (const void *)k_cg32_res<3>;
  int per = 0;
  if (W.res_smem > (size_t)smem ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kResThreads, W.res_smem) !=
          cudaSuccess ||
      per < 1) {
    cudaGetLastError();
    return cudaSuccess;
  }
  A.n = n;
  A.nb = nb;
  A.lanes = L;
  A.warps = warps;
  A.bonds_per_lane = M;
  A.flags = D.flags;
  A.rowptr = D.rowptr;
  A.halo = (const int *)p[0];
  A.nh = (const int *)p[1];
  A.lid = (const uint16_t *)p[2];
  A.words = (unsigned long long *)p[3];
  A.stride = blocks;
  A.status = (int *)(A.words + 3 * (size_t)blocks);
  A.count = (unsigned *)A.status + 1;
  if ((e = cudaMemsetAsync(p[3], 0, bytes[3], s)) != cudaSuccess) return e;
  W.epoch = 0;
  A.z = (float *)p[4];
  A.res = (double *)p[5];
  A.blk = W.blk;
  A.dblk = W.dblk;
  A.blocks = blocks;
  return cudaSuccess;
}

// Newton correction (-K) dx = rhs.  The FP32 solve is tried first; when it
// has not reached the tolerance within kCg32Cap iterations (tangents of
// fractured states are too ill-conditioned for FP32 recurrences), the FP64
// solve takes over from scratch and *use64 is set so that the caller keeps
// FP64 for the rest of the load step.
constexpr int kCg32Cap = 800;

cudaError_t qs_cg(const StepParams &P, const DevPtrs &D, QSWork &W, const double *rhs,
                  double *dx, double tol, int max_iters, int check_every, int *iters,
                  bool *use64, cudaStream_t s) {
  int it32 = 0;
  if (!*use64) {
    bool conv = false;
    cudaError_t e = cudaSuccess;
    int status = 0;
    const int cap = std::min(max_iters, kCg32Cap);
    if (W.kr.blocks > 0) {
      e = qs_cg32_res(P, D, W, rhs, dx, tol, cap, &it32, &conv, &status, s);
      if (e == cudaSuccess && status != 0) {
        if (W.res_only) return cudaErrorTimeout;
        W.kr.blocks = 0;  // the two-launch form from now on
      }
    }
    if (e == cudaSuccess && W.kr.blocks == 0)
      e = qs_cg32(P, D, W, rhs, dx, tol, cap, check_every, &it32, &conv, s);
    if (e != cudaSuccess || conv || max_iters <= kCg32Cap) {
      *iters = it32;
      return e;
    }
    *use64 = true;
  }
  int it64 = 0;
  cudaError_t e = qs_cg64(P, D, W, rhs, dx, tol, max_iters, check_every, &it64, s);
  *iters = it32 + it64;
  return e;
}

// dx = u - u_prev (DIM per node); with fixed_only, 0 on free dofs
template <int DIM>
__global__ void k_qs_bcdiff(int64_t n, const uint8_t *flags, const double *u,
                            const double *uprev, double *dx, bool fixed_only) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int S = DIM == 2 ? 2 : 4;
  for (int c = 0; c < DIM; c++)
    dx[DIM * i + c] =
        (!fixed_only || (flags[i] >> c & 1)) ? u[S * i + c] - uprev[S * i + c] : 0.;
}
__global__ void k_qs_sub(int64_t m, const double *a, const double *b, double *out) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < m) out[k] = a[k] - b[k];
}

cudaError_t qs_bcdiff(const StepParams &P, const DevPtrs &D, const double *u,
                      const double *uprev, double *dx, bool fixed_only, cudaStream_t s) {
  if (P.dim == 2)
    k_qs_bcdiff<2><<<qblk(P.n), 256, 0, s>>>(P.n, D.flags, u, uprev, dx, fixed_only);
  else
    k_qs_bcdiff<3><<<qblk(P.n), 256, 0, s>>>(P.n, D.flags, u, uprev, dx, fixed_only);
  return cudaGetLastError();
}

cudaError_t qs_spmv(const StepParams &P, const DevPtrs &D, const double *blk, const double *dblk,
                    const double *x, double *y, double *part, cudaStream_t s) {
  // part: grp_blocks(n) partials of x.y
  if (P.dim == 2)
    k_cg_dir_spmv<2, false><<<grp_blocks(P.n), 256, 0, s>>>(
        P.n, D.flags, D.rowptr, D.cols, blk, dblk, x, nullptr, nullptr, y, nullptr, nullptr,
        part, nullptr, nullptr);
  else
    k_cg_dir_spmv<3, false><<<grp_blocks(P.n), 256, 0, s>>>(
        P.n, D.flags, D.rowptr, D.cols, blk, dblk, x, nullptr, nullptr, y, nullptr, nullptr,
        part, nullptr, nullptr);
  return cudaGetLastError();
}

cudaError_t qs_sub(int64_t m, const double *a, const double *b, double *out, cudaStream_t s) {
  k_qs_sub<<<qblk(m), 256, 0, s>>>(m, a, b, out);
  return cudaGetLastError();
}

cudaError_t qs_add(const StepParams &P, const double *du, double *u, cudaStream_t s) {
  if (P.dim == 2)
    k_qs_add<2><<<qblk(P.n), 256, 0, s>>>(P.n, du, u);
  else
    k_qs_add<3><<<qblk(P.n), 256, 0, s>>>(P.n, du, u);
  return cudaGetLastError();
}

}  // namespace nlm
