// esqs_internal.h -- launchers of the quasi-static ElasticState solver (esqs.cu).
#pragma once

#include <cstdint>

#include "fd_internal.h"

namespace nlm {

// Partial sums of esqs_dot (the part buffer holds this many doubles).
constexpr int kEsqsDotParts = 512;

// theta (n doubles) and the force density f (S per node) at u.
cudaError_t esqs_force(const StepParams &P, const DevPtrs &D, int S, int mdim, const double *u,
                       double *theta, double *f, cudaStream_t s);
// r = f + b on free dofs, 0 on fixed dofs.
cudaError_t esqs_residual(const StepParams &P, const DevPtrs &D, int S, int mdim,
                          const double *f, const double *b, double *r, cudaStream_t s);
// ocols: original column id of every directed bond
cudaError_t esqs_topology(const StepParams &P, const DevPtrs &D, int *ocols, cudaStream_t s);
// Jacobian blocks (mdim^2 each, nnz + n of them) at u; theta: the dilatations
// at u; bond: 2 mdim doubles per directed bond, sums: 2 mdim + mdim^2 per node
cudaError_t esqs_jacobian(const StepParams &P, const DevPtrs &D, int S, int mdim, int full,
                          const double *u, const double *theta, double eps, const int *ocols,
                          double *bond, double *sums, double *J, cudaStream_t s);
// BiCGSTAB state on the device (sc: slots 0-1 written by the direction launch,
// 2-3 by the shadow launch, by iteration parity).
struct BiScal {
  double rho, alpha, omega, beta, stop2;
  int done, iters;
  int moved;                // x and r are those of this iteration's end already
};
// done: the solve goes on, is over, ends with the x update of this dir launch, or
// sums r.r and rhat.r afresh in it
enum { BI_RUN = 0, BI_DONE = 1, BI_LAST = 2, BI_SUM = 3 };
constexpr int kBiParts = 1216;  // most blocks of a launch (8 per SM)
struct BiArgs {
  int64_t n, m;             // nodes, entries of a vector (S per node)
  const uint8_t *flags;
  const int64_t *rowptr;
  const int *cols;
  const double *J;
  double *r, *rhat, *p[2], *v[2], *s, *t, *x;
  double *part1, *part2, *part3;  // kBiParts, 5 kBiParts and 2 kBiParts doubles
  int blocks;
  BiScal *sc;               // 4
  double tol;               // ||r|| <= tol ||rhs||
  int max_iters;
};
constexpr int kBiGraph = 32;  // iterations per graph launch (even)
int esqs_bicgstab_blocks(int64_t n);
cudaError_t esqs_bicgstab_graph(const BiArgs &B, int mdim, cudaGraphExec_t *out, cudaStream_t s);
// J x = rhs; synchronises.
cudaError_t esqs_bicgstab(const BiArgs &B, cudaGraphExec_t graph, const double *rhs, int *iters,
                          cudaStream_t s);
// out = a x + b y + c z; y or z may be NULL.
cudaError_t esqs_lin3(int64_t m, double a, const double *x, double b, const double *y, double c,
                      const double *z, double *out, cudaStream_t s);
// *out = a . b (device scalar), via kEsqsDotParts partial sums in part.
cudaError_t esqs_dot(int64_t m, const double *a, const double *b, double *part, double *out,
                     cudaStream_t s);

}  // namespace nlm
