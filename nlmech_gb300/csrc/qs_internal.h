// qs_internal.h -- work buffers and launchers of the quasi-static solver.
#pragma once

#include <functional>

#include "fd_internal.h"

namespace nlm {

// The FP32 Krylov solve in one cooperative launch (qs.cu: k_cg32_res).
constexpr int kResHalo = 2048;  // most halo nodes of a block
struct CgRes {
  int64_t n;
  int blocks, nb;          // grid, consecutive nodes of a block
  int lanes, warps, bonds_per_lane;  // lanes per node, warps with nodes, longest share
  uint32_t epoch;          // iteration numbers of this solve start above it
  const uint8_t *flags;
  const int64_t *rowptr;
  const int *halo, *nh;    // kResHalo ids per block, and how many
  const uint16_t *lid;     // per bond: local id of the neighbour
  const double *blk, *dblk, *rhs;
  double *dx;
  float *z;                // DIM per node
  unsigned long long *words;  // 3 x stride: (iteration, FP32 partial) of each block
  int stride, extra;       // extra: arrivals a sum waits for that nobody makes (tests)
  unsigned *count;         // arrivals of this solve
  const double *rr0;       // r.r of the right-hand side
  double tol2;
  int max_iters;
  int *status;
  uint64_t wait_ns;        // bound of each wait
  double *res;
};

struct QSWork {
  double *res;    // residual, DIM per node
  double *dx;     // Newton correction
  double *r, *z, *p, *ap;  // CG vectors
  double *p2;     // second search-direction buffer (iteration parity)
  double *cgpart; // CG partial sums: 3 arrays of qs_cg_stride(n) entries
  double *cgs;    // CG totals on the device (4) and two FP32 step lengths
  unsigned *ticket;  // last-block tickets of the two CG launches (start at 0)
  double *part;   // block partial sums
  double *sc;     // device scalars
  double *blk;    // tangent blocks per bond (3 or 6 doubles)
  double *dblk;   // diagonal blocks per node
  double *res0;   // force at the previous converged state
  // FP32 Krylov solve: tangent copies and CG vectors
  float *blk32, *dblk32, *minv32, *r32, *z32, *p32, *p32b, *ap32, *x32;
  int64_t nnz;
  CgRes kr;         // kr.blocks == 0: two launches per iteration
  size_t res_smem;
  uint32_t epoch;   // iteration numbers used up by earlier solves
  bool res_only;    // a wait that runs out is an error (else: two launches)
};

// Lay out the resident FP32 solve in W.kr (blocks = 0: not available).
cudaError_t qs_res_setup(const StepParams &P, const DevPtrs &D, const int64_t *rowptr_host,
                         QSWork &W, const std::function<cudaError_t(void **, size_t)> &alloc,
                         cudaStream_t s);

// count != NULL: bonds past the critical strain break during the evaluation
// (RNPBond::getBondEF) and the number broken is added to *count.
cudaError_t qs_residual(const StepParams &P, const DevPtrs &D, const double *u, double *res,
                        double *blk, double *dblk, bool assemble, cudaStream_t s,
                        unsigned long long *count = nullptr);
cudaError_t qs_dot(const double *a, const double *b, int64_t m, double *part, double *out,
                   cudaStream_t s);
// use64: in/out, FP64 Krylov solve (set when the FP32 solve did not converge)
cudaError_t qs_cg(const StepParams &P, const DevPtrs &D, QSWork &W, const double *rhs,
                  double *dx, double tol, int max_iters, int check_every, int *iters,
                  bool *use64, cudaStream_t s);
// Entries per partial-sum array of the CG (4 arrays live in QSWork::cgpart).
int64_t qs_cg_stride(int64_t n);
cudaError_t qs_add(const StepParams &P, const double *du, double *u, cudaStream_t s);
cudaError_t qs_bcdiff(const StepParams &P, const DevPtrs &D, const double *u,
                      const double *uprev, double *dx, bool fixed_only, cudaStream_t s);
cudaError_t qs_spmv(const StepParams &P, const DevPtrs &D, const double *blk, const double *dblk,
                    const double *x, double *y, double *part, cudaStream_t s);
cudaError_t qs_sub(int64_t m, const double *a, const double *b, double *out, cudaStream_t s);

}  // namespace nlm
