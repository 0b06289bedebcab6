// esqs_host.cu -- nlm_esqs_*: quasi-static ElasticState
// (QuasiStaticModel<ElasticState>) on the GPU.

#include "fd_handle.h"

// ===========================================================================
// Quasi-static ElasticState (QuasiStaticModel<ElasticState>).  Geometry,
// volumes, m_i, flags and loads come from an FP64 nlm_fd handle (a 1-D mesh
// is held as a 2-D one with y = 0; the material law uses the model's own
// dimension); the state is its displacement buffer u64[cur].

struct nlm_esqs {
  nlm_fd *fd = nullptr;
  nlm_esqs_params prm{};
  int mdim = 2;
  int64_t m = 0, nblocks = 0;
  double *theta = nullptr, *f = nullptr, *body = nullptr, *res = nullptr, *rhs = nullptr;
  double *dx = nullptr, *J = nullptr, *part = nullptr, *sc = nullptr;
  BiArgs bi{};
  cudaGraphExec_t bi_graph = nullptr;
  // Jacobian assembly: per-bond differences, row sums, original column of a bond
  double *bond = nullptr, *sums = nullptr;
  int *ocols = nullptr;
  std::vector<void *> allocs;
  ~nlm_esqs() {
    if (fd && fd->stream) cudaStreamSynchronize(fd->stream);
    if (bi_graph) cudaGraphExecDestroy(bi_graph);
    if (fd) nlm_fd_destroy(fd);  // synchronises and frees the stream first
    for (void *q : allocs) cudaFree(q);
  }
  template <class Tp>
  cudaError_t alloc(Tp **ptr, size_t count_) {
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, count_ * sizeof(Tp) + 16);
    if (e == cudaSuccess) {
      allocs.push_back(q);
      *ptr = static_cast<Tp *>(q);
    }
    return e;
  }
};

namespace {

int esqs_dot_host(nlm_esqs *q, const double *a, const double *b, double *out) {
  cudaStream_t s = q->fd->stream;
  cudaError_t e = esqs_dot(q->m, a, b, q->part, q->sc, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, q->sc, sizeof(double), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return e == cudaSuccess ? NLM_OK : cuda_fail(e, "quasi-static dot product");
}

// f and the residual r = f + b at the current u; *norm = ||r||.
int esqs_eval(nlm_esqs *q, double *norm) {
  nlm_fd *h = q->fd;
  cudaError_t e = esqs_force(h->P, h->D, h->S, q->mdim, h->D.u64[h->cur], q->theta, q->f, h->stream);
  if (e == cudaSuccess) e = esqs_residual(h->P, h->D, h->S, q->mdim, q->f, q->body, q->res, h->stream);
  if (e != cudaSuccess) return cuda_fail(e, "quasi-static residual");
  double rr = 0.;
  int rc = esqs_dot_host(q, q->res, q->res, &rr);
  *norm = std::sqrt(rr);
  return rc;
}

}  // namespace

extern "C" {

int nlm_esqs_create(const nlm_fd_desc *desc, const nlm_esqs_params *prm, nlm_esqs **out) {
  if (!desc || !prm || !out) return fail(NLM_ERR_INVALID, "null argument");
  *out = nullptr;
  if (desc->material.kind != NLM_MAT_ELASTIC_STATE)
    return fail(NLM_ERR_UNSUPPORTED, "QuasiStaticModel is instantiated for ElasticState");
  if (desc->dim < 1 || desc->dim > 3) return fail(NLM_ERR_INVALID, "dimension must be 1, 2 or 3");
  if (desc->dim == 1 && !(desc->material.E > 0.))
    return fail(NLM_ERR_INVALID, "1-D ElasticState needs E");
  if (prm->max_iters < 0 || !(prm->tol > 0.) || !(prm->perturbation > 0.) ||
      prm->lin_max_iters < 1 || !(prm->lin_tol > 0.) || !(prm->dt > 0.))
    return fail(NLM_ERR_INVALID, "bad solver parameters");
  for (int c = 0; c < desc->n_cracks; c++)
    if (desc->cracks && desc->cracks[c].timed)
      return fail(NLM_ERR_UNSUPPORTED, "the quasi-static solver takes pre-cracks only");
  nlm_fd_desc d = *desc;
  d.precision = NLM_PREC_FP64;
  d.scheme = NLM_VELOCITY_VERLET;
  d.decomposition = NLM_DECOMP_THREAD;
  d.dt = prm->dt;
  d.material.es_sc = 0.;  // no bond breaks in QuasiStaticModel
  std::vector<double> x1;
  if (desc->dim == 1) {
    // a 1-D mesh as a 2-D one: nodes (x, 0, 0); the 2-D constants are unused
    d.dim = 2;
    x1.assign(3 * (size_t)desc->n_nodes, 0.);
    for (int64_t i = 0; i < desc->n_nodes && desc->x; i++) x1[3 * i] = desc->x[3 * i];
    d.x = x1.data();
    if (!(d.material.K > 0.)) d.material.K = 1.;
    if (!(d.material.G > 0.)) d.material.G = 1.;
  }
  nlm_esqs *q = new nlm_esqs();
  int rc = create_model(&d, &q->fd, false);
  if (rc) {
    delete q;
    return rc;
  }
  q->prm = *prm;
  q->mdim = desc->dim;
  nlm_fd *h = q->fd;
  q->m = (int64_t)h->S * h->n;
  q->nblocks = h->nnz + h->n;
  cudaError_t e = q->alloc(&q->theta, h->n);
  BiArgs &bi = q->bi;
  for (double **ptr : {&q->f, &q->body, &q->res, &q->rhs, &q->dx, &bi.r, &bi.rhat, &bi.p[0],
                       &bi.p[1], &bi.v[0], &bi.v[1], &bi.s, &bi.t})
    if (e == cudaSuccess) e = q->alloc(ptr, q->m);
  if (e == cudaSuccess) e = q->alloc(&bi.part1, kBiParts);
  if (e == cudaSuccess) e = q->alloc(&bi.part2, 5 * kBiParts);
  if (e == cudaSuccess) e = q->alloc(&bi.part3, 2 * kBiParts);
  if (e == cudaSuccess) e = q->alloc(&bi.sc, 4);
  const size_t md = (size_t)q->mdim;
  if (e == cudaSuccess) e = q->alloc(&q->J, md * md * q->nblocks);
  if (e == cudaSuccess) e = q->alloc(&q->bond, 2 * md * (size_t)h->nnz);
  if (e == cudaSuccess) e = q->alloc(&q->sums, (2 * md + md * md) * (size_t)h->n);
  if (e == cudaSuccess) e = q->alloc(&q->ocols, (size_t)h->nnz);
  if (e == cudaSuccess) e = esqs_topology(h->P, h->D, q->ocols, h->stream);
  if (e == cudaSuccess) e = q->alloc(&q->part, kEsqsDotParts);
  if (e == cudaSuccess) e = q->alloc(&q->sc, 1);
  bi.n = h->n;
  bi.m = q->m;
  bi.flags = h->D.flags;
  bi.rowptr = h->D.rowptr;
  bi.cols = h->D.cols;
  bi.J = q->J;
  bi.x = q->dx;
  bi.tol = prm->lin_tol;
  bi.max_iters = prm->lin_max_iters;
  bi.blocks = esqs_bicgstab_blocks(h->n);
  if (e == cudaSuccess) e = cudaMemsetAsync(q->body, 0, sizeof(double) * q->m, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) {
    delete q;
    return cuda_fail(e, "quasi-static buffers");
  }
  h->started = true;  // no explicit step-0 evaluation
  *out = q;
  return NLM_OK;
}

int nlm_esqs_destroy(nlm_esqs *q) {
  delete q;
  return NLM_OK;
}

int nlm_esqs_solve(nlm_esqs *q, int nsteps, int *newton_iters, int *lin_iters,
                   double *final_res) {
  if (!q || nsteps < 0) return fail(NLM_ERR_INVALID, "bad arguments");
  nlm_fd *h = q->fd;
  cudaStream_t s = h->stream;
  double *u = h->D.u64[h->cur];
  const double eps = q->prm.perturbation * h->P.h;
  double res = 0.;
  int rc;
  for (int k = 0; k < nsteps; k++) {
    // QuasiStaticModel::solver (:526-594): time = n dt, force loading (added
    // to the body force, fLoading.cpp:268-275), displacement loading
    h->step++;
    h->time = (double)h->step * q->prm.dt;
    if (h->n_fbc_nodes > 0) {
      if ((rc = apply_fbc(h, h->time))) return rc;
      cudaError_t e = esqs_lin3(q->m, 1., q->body, 1., h->D.fext, 0., nullptr, q->body, s);
      if (e != cudaSuccess) return cuda_fail(e, "quasi-static body force");
    }
    if ((rc = apply_bc(h, h->time))) return rc;
    if ((rc = esqs_eval(q, &res))) return rc;
    const double r0 = res;
    int it = 0, li_total = 0;
    auto converged = [&]() {
      return q->prm.tol_relative ? (r0 == 0. || res / r0 < q->prm.tol) : res < q->prm.tol;
    };
    while (!converged() && it < q->prm.max_iters) {
      // theta is esqs_eval's, at the current u
      cudaError_t e = esqs_jacobian(h->P, h->D, h->S, q->mdim, q->prm.jacobian, u, q->theta, eps,
                                    q->ocols, q->bond, q->sums, q->J, s);
      if (e == cudaSuccess) e = esqs_lin3(q->m, -1., q->res, 0., nullptr, 0., nullptr, q->rhs, s);
      if (e != cudaSuccess) return cuda_fail(e, "quasi-static Jacobian");
      int li = 0;
      if (!q->bi_graph) e = esqs_bicgstab_graph(q->bi, q->mdim, &q->bi_graph, s);
      if (e == cudaSuccess) e = esqs_bicgstab(q->bi, q->bi_graph, q->rhs, &li, s);
      if (e != cudaSuccess) return cuda_fail(e, "quasi-static linear solve");
      li_total += li;
      e = esqs_lin3(q->m, 1., u, 1., q->dx, 0., nullptr, u, s);
      if (e != cudaSuccess) return cuda_fail(e, "quasi-static update");
      if ((rc = esqs_eval(q, &res))) return rc;
      it++;
    }
    if (newton_iters) newton_iters[k] = it;
    if (lin_iters) lin_iters[k] = li_total;
  }
  if (final_res) *final_res = res;
  return NLM_OK;
}

int nlm_esqs_get_state(nlm_esqs *q, double *u, double *force) {
  if (!q) return fail(NLM_ERR_INVALID, "null handle");
  nlm_fd *h = q->fd;
  if (u) {
    int rc = nlm_fd_get_state(h, u, nullptr, nullptr);
    if (rc) return rc;
  }
  if (force) {
    const int64_t n = h->n;
    std::vector<double> fi((size_t)q->m), vol(n);
    NLM_CUDA(cudaMemcpyAsync(fi.data(), q->f, sizeof(double) * q->m, cudaMemcpyDeviceToHost, h->stream));
    NLM_CUDA(cudaMemcpyAsync(vol.data(), h->D.vol64, sizeof(double) * n, cudaMemcpyDeviceToHost, h->stream));
    NLM_CUDA(cudaStreamSynchronize(h->stream));
    for (int64_t i = 0; i < n; i++) {
      const int64_t o = h->perm[i];
      for (int d = 0; d < 3; d++) {
        const double fd = (d < h->S && d < q->mdim) ? fi[(size_t)h->S * i + d] : 0.;
        force[3 * o + d] = fd * vol[i];
      }
    }
  }
  return NLM_OK;
}

}  // extern "C"

