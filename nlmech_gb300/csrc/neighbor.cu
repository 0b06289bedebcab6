// neighbor.cu -- uniform-grid horizon neighbour search and bond-store setup.
//
// Replaces geometry::Neighbor (src/geometry/neighbor.cpp:24-92).  The
// reference tests every pair (O(N^2)); here nodes are binned into cells of
// edge >= horizon + 1e-10, sorted by the Morton code of their cell, and each
// node tests only the 3^dim surrounding cells.  The predicate is the
// reference's, evaluated in FP64 with separately rounded operations:
//   definitelyLessThan(|x_i - x_j|, horizon + 1e-10)   (neighbor.cpp:81-82)
// so the sets are identical.  Rows are then ordered by ascending original id,
// the order the reference's j-loop produces.
//
// Compiled with --fmad=false.

#include <algorithm>
#include <climits>
#include <cmath>
#include <cub/cub.cuh>

#include "fd_internal.h"
#include "neighbor.h"

namespace nlm {

__device__ __forceinline__ uint64_t spread3(uint64_t v) {  // 21 bits -> every 3rd bit
  v &= 0x1fffffull;
  v = (v | v << 32) & 0x1f00000000ffffull;
  v = (v | v << 16) & 0x1f0000ff0000ffull;
  v = (v | v << 8) & 0x100f00f00f00f00full;
  v = (v | v << 4) & 0x10c30c30c30c30c3ull;
  v = (v | v << 2) & 0x1249249249249249ull;
  return v;
}

__device__ __forceinline__ void cell_of(const Grid &g, const double *p, int64_t c[3]) {
  for (int d = 0; d < 3; d++) {
    int64_t k = (int64_t)floor((p[d] - g.lo[d]) / g.cs);
    c[d] = k < 0 ? 0 : (k >= g.nc[d] ? g.nc[d] - 1 : k);
  }
}

// keys: Morton code of the cell (with the specimen id above it); values:
// original node id.
__global__ void k_cell_keys(int64_t n, const double *x, Grid g, const int *specimen,
                            uint64_t *keys, int *vals) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t c[3];
  cell_of(g, x + 3 * i, c);
  uint64_t m = spread3((uint64_t)c[0]) | (spread3((uint64_t)c[1]) << 1) |
               (spread3((uint64_t)c[2]) << 2);
  (void)specimen;
  keys[i] = m;
  vals[i] = (int)i;
}

// Sorted positions (S doubles per node, and in FP32 relative to the grid's
// corner) and the linear cell id of each node.
__global__ void k_gather_sorted(int64_t n, int S, const double *x, const int *perm, Grid g,
                                double *pos, float4 *pf, int64_t *cell) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double *p = x + 3 * (int64_t)perm[i];
  for (int d = 0; d < S; d++) pos[(int64_t)S * i + d] = d < 3 ? p[d] : 0.;
  pf[i] = make_float4((float)(p[0] - g.lo[0]), (float)(p[1] - g.lo[1]),
                      S > 2 ? (float)(p[2] - g.lo[2]) : 0.f, 0.f);
  int64_t c[3];
  cell_of(g, p, c);
  cell[i] = (c[2] * g.nc[1] + c[1]) * g.nc[0] + c[0];
}

__global__ void k_cell_ranges(int64_t n, const int64_t *cell, int64_t *cbeg, int64_t *cend) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t c = cell[i];
  if (i == 0 || cell[i - 1] != c) cbeg[c] = i;
  if (i == n - 1 || cell[i + 1] != c) cend[c] = i + 1;
}

__device__ __forceinline__ bool within(const double *a, const double *b, double rad) {
  // util::Point3::dist (point.h:165-169) with this = x_i, argument = x_j
  const double dx = __dsub_rn(a[0], b[0]), dy = __dsub_rn(a[1], b[1]),
               dz = __dsub_rn(a[2], b[2]);
  const double s = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  return dLT(__dsqrt_rn(s), rad);
}

// Squared FP32 distances (coordinates relative to the grid's corner) that decide
// the predicate without FP64: below in2 it certainly holds, above out2 it
// certainly does not, whatever the FP32 rounding; between them (and for a NaN)
// within() decides.  The FP64 pipe was the bound: a square root and two dozen
// FP64 operations per candidate (350,000 nodes, 60 neighbours: 313 us for the
// counts, the pipe 80 % busy; 111 us now.)
struct NearBand {
  float in2, out2;
};
static NearBand near_band(const Grid &g) {
  double ext = 0.;
  for (int d = 0; d < 3; d++) ext = std::max(ext, g.nc[d] * g.cs);
  // dLT(r, rad) <=> r < rad (1 - 1e-5) up to FP64 rounding; a coordinate
  // difference is good to 2^-23 ext, three of them and the FP32 sum of squares
  // to less than 4 times that plus 1e-6 of the distance
  const double r = g.rad * (1. - 1e-5), e = 4. * std::ldexp(ext, -23) + 2e-6 * g.rad;
  NearBand b;
  b.in2 = r > e ? (float)((r - e) * (r - e) * (1. - 1e-6)) : -1.f;
  b.out2 = (float)((r + e) * (r + e) * (1. + 1e-6));
  return b;
}

// FILL pass.  ROWS_ORIG: rows of the caller's node ids at rowptr[original id];
// otherwise rows of internal ids at rowptr[i].  Rows
// are left in cell order (k_sort_rows orders them).  Counting: count[i], or count[original id] with ROWS_ORIG.
template <bool FILL, bool ROWS_ORIG>
__global__ void __launch_bounds__(128)
    k_neighbors(int64_t n, int S, const double *pos, const float4 *pf, NearBand nb,
                const int64_t *cell, Grid g, const int64_t *cbeg, const int64_t *cend,
                const int *perm, int64_t *count, const int64_t *rowptr, int *cols, int *err) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 pi = pf[i];
  const int64_t ci = cell[i];
  int64_t c[3] = {ci % g.nc[0], (ci / g.nc[0]) % g.nc[1], ci / (g.nc[0] * g.nc[1])};
  int64_t cnt = 0;
  const int64_t row0 = FILL ? rowptr[ROWS_ORIG ? perm[i] : i] : 0;
  int *row = FILL ? cols + row0 : nullptr;
  for (int64_t dz = -1; dz <= 1; dz++) {
    const int64_t z = c[2] + dz;
    if (z < 0 || z >= g.nc[2]) continue;
    for (int64_t dy = -1; dy <= 1; dy++) {
      const int64_t y = c[1] + dy;
      if (y < 0 || y >= g.nc[1]) continue;
      for (int64_t dx = -1; dx <= 1; dx++) {
        const int64_t x = c[0] + dx;
        if (x < 0 || x >= g.nc[0]) continue;
        const int64_t cc = (z * g.nc[1] + y) * g.nc[0] + x;
        const int64_t b = cbeg[cc], e = cend[cc];
        for (int64_t j = b; j < e; j++) {
          if (j == i) continue;
          const float4 pj = __ldg(pf + j);
          const float fx = pi.x - pj.x, fy = pi.y - pj.y, fz = pi.z - pj.z;
          const float s = fx * fx + fy * fy + fz * fz;
          bool near = s < nb.in2;
          if (!near && !(s > nb.out2)) {
            const double xi[3] = {pos[S * i], pos[S * i + 1], S > 2 ? pos[S * i + 2] : 0.};
            const double xj[3] = {pos[S * j], pos[S * j + 1], S > 2 ? pos[S * j + 2] : 0.};
            near = within(xi, xj, g.rad);
          }
          if (near) {
            if (FILL) row[cnt] = ROWS_ORIG ? perm[j] : (int)j;
            cnt++;
          }
        }
      }
    }
  }
  if (!FILL) {
    count[ROWS_ORIG ? perm[i] : i] = cnt;
    if (cnt > kMaxRow) atomicExch(err, DEVERR_ROW_TOO_LONG);
    return;
  }
}

// Order each row by its entries (KEY_PERM: by perm of them): a warp per row
// ranks the entries, which are distinct, against all keys in shared memory.
// With one thread per row inserting, the row pass took 594 us (350,000 rows of
// 60), 186 + 154 us now.
template <bool KEY_PERM>
__global__ void __launch_bounds__(128)
    k_sort_rows(int64_t n, const int64_t *rowptr, const int *perm, int *cols) {
  __shared__ __align__(16) int keys[4][kMaxRow + 4];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = blockIdx.x * 4ll + w;
  if (i >= n) return;
  const int64_t r0 = rowptr[i];
  const int len = (int)(rowptr[i + 1] - r0), len4 = (len + 3) & ~3;
  int *row = cols + r0, *key = keys[w];
  int v[kMaxRow / 32];
#pragma unroll 2
  for (int u = 0, k = lane; k < len; u++, k += 32) {
    v[u] = row[k];
    key[k] = KEY_PERM ? perm[v[u]] : v[u];
  }
  for (int k = len + lane; k < len4; k += 32) key[k] = INT_MAX;
  __syncwarp();
  for (int u = 0, k = lane; k < len; u += 2, k += 64) {
    const int a = key[k], b = k + 32 < len ? key[k + 32] : INT_MAX;
    int ra = 0, rb = 0;
    for (int q = 0; q < len4; q += 4) {
      const int4 t = *reinterpret_cast<const int4 *>(key + q);
      ra += (t.x < a) + (t.y < a) + (t.z < a) + (t.w < a);
      rb += (t.x < b) + (t.y < b) + (t.z < b) + (t.w < b);
    }
    row[ra] = v[u];
    if (k + 32 < len) row[rb] = v[u + 1];
  }
}

__global__ void k_sell_width(int64_t n, const int64_t *rowptr, int *width) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int len = (int)(rowptr[i + 1] - rowptr[i]);
  atomicMax(width + (i >> 5), len);
}

// Sliced ELL, 32 rows per slice, entries interleaved in groups of four: entry
// k of lane l sits at slice_base + (k/4)*128 + 4l + k%4, so a thread fetches
// four neighbour ids with one 16-byte load and a warp's load is 512
// contiguous bytes.  Slice widths are multiples of 4; pads are -1.
__global__ void k_sell_fill(int64_t n, int64_t nslices, const int64_t *rowptr, const int *cols,
                            const int64_t *sell_ptr, const int *width, int *sell_cols) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= nslices * 32) return;
  const int64_t s = t >> 5;
  const int lane = (int)(t & 31);
  const int64_t i = t;
  const int w = width[s];
  const int64_t base = sell_ptr[s] + 4 * lane;
  const int64_t r0 = i < n ? rowptr[i] : 0;
  const int len = i < n ? (int)(rowptr[i + 1] - r0) : 0;
  for (int k = 0; k < w; k++)
    sell_cols[base + (int64_t)(k >> 2) * 128 + (k & 3)] = k < len ? cols[r0 + k] : -1;
}

// Pre-crack bits (geometry::Fracture ctor, src/geometry/fracture.cpp:20-160;
// inp::EdgeCrack predicates, src/inp/decks/fractureDeck.h:115-186).
__device__ bool pt_outside(const nlm_crack &c, const double *p) {
  if (c.orientation == -1) return dLT(p[1], c.pb[1]) || dGT(p[1], c.pt[1]);
  if (c.orientation == 1) return dLT(p[0], c.pb[0]) || dGT(p[0], c.pt[0]);
  if (c.orientation == 0) {
    const double px = __dsub_rn(p[0], c.pb[0]), py = __dsub_rn(p[1], c.pb[1]);
    const double tx = __dsub_rn(c.pt[0], c.pb[0]), ty = __dsub_rn(c.pt[1], c.pb[1]);
    const double ct = cos(c.theta), st = sin(c.theta);
    const double pmx = __dadd_rn(__dmul_rn(ct, px), __dmul_rn(st, py));
    const double ptx = __dadd_rn(__dmul_rn(ct, tx), __dmul_rn(st, ty));
    return dLT(pmx, 0.0) || dGT(pmx, ptx);
  }
  return true;
}
__device__ bool pt_left(const nlm_crack &c, const double *p) {
  const double a = __dmul_rn(
      0.5, __dsub_rn(__dmul_rn(__dsub_rn(c.pt[0], c.pb[0]), __dsub_rn(p[1], c.pb[1])),
                     __dmul_rn(__dsub_rn(p[0], c.pb[0]), __dsub_rn(c.pt[1], c.pb[1]))));
  return !dLT(a, 0.0);
}
__device__ bool plane_cuts(const nlm_crack &c, const double *a, const double *b) {
  const bool sa = a[2] < c.z0, sb = b[2] < c.z0;
  if (sa == sb) return false;
  const double t = (c.z0 - a[2]) / (b[2] - a[2]);
  const double px = a[0] + t * (b[0] - a[0]);
  const double py = a[1] + t * (b[1] - a[1]);
  return px >= c.lo[0] && px <= c.hi[0] && py >= c.lo[1] && py <= c.hi[1];
}

__global__ void k_precrack(int64_t n, int64_t off, int S, const double *pos,
                           const int64_t *rowptr, const int *cols, nlm_crack ck, int64_t npad,
                           uint32_t *bits) {
  const int64_t i = off + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= off + n) return;
  const double xi[3] = {pos[S * i], pos[S * i + 1], S > 2 ? pos[S * i + 2] : 0.};
  const int64_t r0 = rowptr[i], r1 = rowptr[i + 1];
  if (ck.kind == NLM_CRACK_PLANE) {
    for (int64_t k = r0; k < r1; k++) {
      const int64_t j = cols[k];
      const double xj[3] = {pos[S * j], pos[S * j + 1], S > 2 ? pos[S * j + 2] : 0.};
      if (plane_cuts(ck, xi, xj)) {
        const int kk = (int)(k - r0);
        bits[(int64_t)(kk >> 5) * npad + i] |= 1u << (kk & 31);
      }
    }
    return;
  }
  if (pt_outside(ck, xi)) return;
  const bool left = pt_left(ck, xi);
  for (int64_t k = r0; k < r1; k++) {
    const int64_t j = cols[k];
    const double xj[3] = {pos[S * j], pos[S * j + 1], S > 2 ? pos[S * j + 2] : 0.};
    const bool modify = !pt_outside(ck, xj);
    const bool other = left ? !pt_left(ck, xj) : pt_left(ck, xj);
    if (other && modify) {
      const int kk = (int)(k - r0);
      bits[(int64_t)(kk >> 5) * npad + i] |= 1u << (kk & 31);
    }
  }
}

// ---------------------------------------------------------------------------
// host driver

#define NB_CHECK(call)                          \
  do {                                          \
    cudaError_t _e = (call);                    \
    if (_e != cudaSuccess) return _e;           \
  } while (0)

static unsigned blocks(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

static Grid grid_of(const double lo[3], const double hi[3], double horizon) {
  Grid g;
  g.rad = horizon + 1.0E-10;
  g.cs = g.rad * (1.0 + 1e-7);
  for (int d = 0; d < 3; d++) {
    g.lo[d] = lo[d];
    const int64_t k = (int64_t)((hi[d] - lo[d]) / g.cs) + 1;
    g.nc[d] = k < 1 ? 1 : k;
  }
  return g;
}

Grid make_grid(int dim, int64_t n, const double *x, double horizon) {
  double lo[3] = {0., 0., 0.}, hi[3] = {0., 0., 0.};
  for (int d = 0; d < 3 && n > 0; d++) {
    lo[d] = 1e300;
    hi[d] = -1e300;
    for (int64_t i = 0; i < n; i++) {
      lo[d] = x[3 * i + d] < lo[d] ? x[3 * i + d] : lo[d];
      hi[d] = x[3 * i + d] > hi[d] ? x[3 * i + d] : hi[d];
    }
  }
  (void)dim;
  return grid_of(lo, hi, horizon);
}

// Bounding box and finiteness of the coordinates, one line of 8 doubles per
// block: lo, hi, bad (0 or 1).
constexpr int kBoxBlocks = 304;
__global__ void __launch_bounds__(256) k_bbox(int64_t n, const double *x, double *out) {
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  int bad = 0;
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += 256ll * gridDim.x)
    for (int d = 0; d < 3; d++) {
      const double v = x[3 * i + d];
      if (!isfinite(v)) bad = 1;
      if (v < lo[d]) lo[d] = v;
      if (v > hi[d]) hi[d] = v;
    }
  __shared__ double sh[6][8];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  for (int d = 0; d < 3; d++) {
    for (int o = 16; o > 0; o >>= 1) {
      const double a = __shfl_xor_sync(0xffffffffu, lo[d], o);
      const double b = __shfl_xor_sync(0xffffffffu, hi[d], o);
      if (a < lo[d]) lo[d] = a;
      if (b > hi[d]) hi[d] = b;
    }
    if (l == 0) {
      sh[d][w] = lo[d];
      sh[3 + d][w] = hi[d];
    }
  }
  bad = __syncthreads_or(bad);
  if (threadIdx.x < 6) {
    double v = sh[threadIdx.x][0];
    for (int q = 1; q < 8; q++) {
      const double a = sh[threadIdx.x][q];
      v = threadIdx.x < 3 ? (a < v ? a : v) : (a > v ? a : v);
    }
    out[8 * blockIdx.x + threadIdx.x] = v;
  }
  if (threadIdx.x == 6) out[8 * blockIdx.x + 6] = bad;
}

cudaError_t build_neighbors(NeighborBuild &nb, int dim, int64_t n, const double *d_x,
                            const Grid &g, int S, cudaStream_t s, std::string &why,
                            bool rows_by_orig) {
  nb.n = n;
  nb.S = S;
  const int bs = 256;
  uint64_t *keys = nullptr, *keys2 = nullptr;
  int *vals = nullptr;
  int *err = nullptr;
  float4 *pf = nullptr;
  int64_t *cell = nullptr, *cbeg = nullptr, *cend = nullptr, *cnt = nullptr;
  void *tmp = nullptr;
  size_t tmpb = 0;
  const int64_t ncell = g.nc[0] * g.nc[1] * g.nc[2];
  const NearBand band = near_band(g);
  cudaError_t e = cudaSuccess;
  auto cleanup = [&]() {
    cudaFree(keys); cudaFree(keys2); cudaFree(vals); cudaFree(err); cudaFree(cell);
    cudaFree(cbeg); cudaFree(cend); cudaFree(cnt); cudaFree(tmp); cudaFree(pf);
  };
#define NB_TRY(call)             \
  do {                           \
    e = (call);                  \
    if (e != cudaSuccess) {      \
      cleanup();                 \
      return e;                  \
    }                            \
  } while (0)
  NB_TRY(cudaMalloc(&keys, sizeof(uint64_t) * (n + 1)));
  NB_TRY(cudaMalloc(&keys2, sizeof(uint64_t) * (n + 1)));
  NB_TRY(cudaMalloc(&vals, sizeof(int) * (n + 1)));
  NB_TRY(cudaMalloc(&nb.perm, sizeof(int) * (n + 1)));
  NB_TRY(cudaMalloc(&err, sizeof(int)));
  NB_TRY(cudaMemsetAsync(err, 0, sizeof(int), s));
  if (n > 0) {
    k_cell_keys<<<blocks(n, bs), bs, 0, s>>>(n, d_x, g, nullptr, keys, vals);
    NB_TRY(cudaGetLastError());
    NB_TRY(cub::DeviceRadixSort::SortPairs(nullptr, tmpb, keys, keys2, vals, nb.perm, (int)n, 0,
                                           64, s));
    NB_TRY(cudaMalloc(&tmp, tmpb));
    NB_TRY(cub::DeviceRadixSort::SortPairs(tmp, tmpb, keys, keys2, vals, nb.perm, (int)n, 0, 64,
                                           s));
    cudaFree(tmp);
    tmp = nullptr;
  }
  NB_TRY(cudaMalloc(&nb.pos, sizeof(double) * S * (n + 1)));
  NB_TRY(cudaMalloc(&pf, sizeof(float4) * (n + 1)));
  NB_TRY(cudaMalloc(&cell, sizeof(int64_t) * (n + 1)));
  NB_TRY(cudaMalloc(&cbeg, sizeof(int64_t) * ncell));
  NB_TRY(cudaMalloc(&cend, sizeof(int64_t) * ncell));
  NB_TRY(cudaMemsetAsync(cbeg, 0, sizeof(int64_t) * ncell, s));
  NB_TRY(cudaMemsetAsync(cend, 0, sizeof(int64_t) * ncell, s));
  NB_TRY(cudaMalloc(&cnt, sizeof(int64_t) * (n + 1)));
  NB_TRY(cudaMalloc(&nb.rowptr, sizeof(int64_t) * (n + 1)));
  if (n > 0) {
    k_gather_sorted<<<blocks(n, bs), bs, 0, s>>>(n, S, d_x, nb.perm, g, nb.pos, pf, cell);
    NB_TRY(cudaGetLastError());
    k_cell_ranges<<<blocks(n, bs), bs, 0, s>>>(n, cell, cbeg, cend);
    NB_TRY(cudaGetLastError());
    k_neighbors<false, false><<<blocks(n, 128), 128, 0, s>>>(n, S, nb.pos, pf, band, cell, g,
                                                             cbeg, cend, nb.perm, cnt, nullptr,
                                                             nullptr, err);
    NB_TRY(cudaGetLastError());
    int herr = 0;
    NB_TRY(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    NB_TRY(cudaStreamSynchronize(s));
    if (herr == DEVERR_ROW_TOO_LONG) {
      why = "a neighbour row exceeds the supported maximum";
      cleanup();
      return cudaErrorInvalidValue;
    }
    NB_TRY(cudaMemsetAsync(cnt + n, 0, sizeof(int64_t), s));
    NB_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tmpb, cnt, nb.rowptr, n + 1, s));
    NB_TRY(cudaMalloc(&tmp, tmpb));
    NB_TRY(cub::DeviceScan::ExclusiveSum(tmp, tmpb, cnt, nb.rowptr, n + 1, s));
  } else {
    NB_TRY(cudaMemsetAsync(nb.rowptr, 0, sizeof(int64_t), s));
  }
  NB_TRY(cudaMemcpyAsync(&nb.nnz, nb.rowptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  NB_TRY(cudaStreamSynchronize(s));
  NB_TRY(cudaMalloc(&nb.cols, sizeof(int) * (nb.nnz + 1)));
  if (n > 0) {
    k_neighbors<true, false><<<blocks(n, 128), 128, 0, s>>>(n, S, nb.pos, pf, band, cell, g,
                                                            cbeg, cend, nb.perm, nullptr,
                                                            nb.rowptr, nb.cols, err);
    // by ascending original id (the reference's order), or by internal index
    (rows_by_orig ? k_sort_rows<true> : k_sort_rows<false>)<<<blocks(n, 4), 128, 0, s>>>(
        n, nb.rowptr, nb.perm, nb.cols);
    NB_TRY(cudaGetLastError());
  }
  NB_TRY(cudaStreamSynchronize(s));
  cleanup();
  return cudaSuccess;
#undef NB_TRY
}

cudaError_t build_sell(int64_t n, const int64_t *rowptr, const int *cols, SellStore &st,
                       cudaStream_t s) {
  const int bs = 256;
  st.nslices = (n + 31) / 32;
  NB_CHECK(cudaMalloc(&st.width, sizeof(int) * (st.nslices + 1)));
  NB_CHECK(cudaMemsetAsync(st.width, 0, sizeof(int) * (st.nslices + 1), s));
  if (n > 0) {
    k_sell_width<<<blocks(n, bs), bs, 0, s>>>(n, rowptr, st.width);
    NB_CHECK(cudaGetLastError());
  }
  std::vector<int> w(st.nslices);
  NB_CHECK(cudaMemcpyAsync(w.data(), st.width, sizeof(int) * st.nslices, cudaMemcpyDeviceToHost, s));
  NB_CHECK(cudaStreamSynchronize(s));
  std::vector<int64_t> ptr(st.nslices + 1, 0);
  st.maxw = 0;
  for (int64_t k = 0; k < st.nslices; k++) {
    st.maxw = w[k] > st.maxw ? w[k] : st.maxw;
    w[k] = (w[k] + 3) & ~3;
    ptr[k + 1] = ptr[k] + 32 * (int64_t)w[k];
  }
  NB_CHECK(cudaMemcpyAsync(st.width, w.data(), sizeof(int) * st.nslices, cudaMemcpyHostToDevice, s));
  st.entries = ptr[st.nslices];
  NB_CHECK(cudaMalloc(&st.ptr, sizeof(int64_t) * (st.nslices + 1)));
  NB_CHECK(cudaMemcpyAsync(st.ptr, ptr.data(), sizeof(int64_t) * (st.nslices + 1),
                           cudaMemcpyHostToDevice, s));
  NB_CHECK(cudaMalloc(&st.cols, sizeof(int) * (st.entries + 1)));
  if (n > 0) {
    k_sell_fill<<<blocks(st.nslices * 32, bs), bs, 0, s>>>(n, st.nslices, rowptr, cols, st.ptr,
                                                           st.width, st.cols);
    NB_CHECK(cudaGetLastError());
  }
  NB_CHECK(cudaStreamSynchronize(s));
  return cudaSuccess;
}

cudaError_t apply_precrack(int64_t n, int S, const double *pos, const int64_t *rowptr,
                           const int *cols, const nlm_crack &ck, int64_t npad, uint32_t *bits,
                           cudaStream_t s, int64_t off) {
  if (n == 0) return cudaSuccess;
  k_precrack<<<blocks(n, 128), 128, 0, s>>>(n, off, S, pos, rowptr, cols, ck, npad, bits);
  return cudaGetLastError();
}

__global__ void k_offset_cols(int64_t nnz, int *cols, int off) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < nnz) cols[k] += off;
}
__global__ void k_offset_rowptr(int64_t n, int64_t *rowptr, int64_t off) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < n) rowptr[k] += off;
}

cudaError_t offset_cols(int64_t nnz, int *cols, int off, cudaStream_t s) {
  if (nnz == 0) return cudaSuccess;
  k_offset_cols<<<blocks(nnz, 256), 256, 0, s>>>(nnz, cols, off);
  return cudaGetLastError();
}
cudaError_t offset_rowptr(int64_t n, int64_t *rowptr, int64_t off, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_offset_rowptr<<<blocks(n, 256), 256, 0, s>>>(n, rowptr, off);
  return cudaGetLastError();
}

// ---- the search on its own ------------------------------------------------------
// Rows in the caller's ids and order straight from the device: the bounding box
// and the finiteness check, the cell sort, the counts, their scan and the rows
// are kernels, with one arena for everything but the rows.  (Before, each of
// the two calls a caller makes sorted and filled in the internal order,
// downloaded the rows and permuted them on one host thread: 42-51 ms for
// 350,000 nodes and 21 million entries, 3.8 ms now, half of it the 84 MB of rows
// into the caller's memory.)

NeighborSearch::~NeighborSearch() {
  cudaFree(arena);
  cudaFree(cols);
  if (s) cudaStreamDestroy(s);
}

cudaError_t search_neighbors(NeighborSearch &R, int64_t n, const double *x, double horizon,
                             bool want_cols, std::string &why) {
  cudaError_t e = cudaSuccess;
  if (!R.s) e = cudaStreamCreateWithFlags(&R.s, cudaStreamNonBlocking);
  cudaStream_t s = R.s;
  R.n = n;
  size_t sort_b = 0, scan_b = 0;
  if (e == cudaSuccess)
    e = cub::DeviceRadixSort::SortPairs(nullptr, sort_b, (const uint64_t *)nullptr,
                                        (uint64_t *)nullptr, (const int *)nullptr, (int *)nullptr,
                                        (int)n, 0, 64, s);
  if (e == cudaSuccess)
    e = cub::DeviceScan::ExclusiveSum(nullptr, scan_b, (const int64_t *)nullptr,
                                      (int64_t *)nullptr, n + 1, s);
  if (e != cudaSuccess) return e;
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t tmp_b = std::max(sort_b, scan_b);
  // x, keys (2), values, perm, pos, pf, cell, count, rowptr, box, err, temp
  const size_t sz[13] = {up(24 * n),      up(8 * n),  up(8 * n),       up(4 * n),       up(4 * n),
                         up(32 * n),      up(16 * n), up(8 * n),       up(8 * (n + 1)),
                         up(8 * (n + 1)), up(64 * kBoxBlocks), up(sizeof(int)), up(tmp_b)};
  size_t total = 0, at[13];
  for (int k = 0; k < 13; k++) {
    at[k] = total;
    total += sz[k];
  }
  if ((e = cudaMalloc(&R.arena, total)) != cudaSuccess) return e;
  char *base = static_cast<char *>(R.arena);
  double *dx = (double *)(base + at[0]), *pos = (double *)(base + at[5]);
  uint64_t *keys = (uint64_t *)(base + at[1]), *keys2 = (uint64_t *)(base + at[2]);
  int *vals = (int *)(base + at[3]), *perm = (int *)(base + at[4]);
  float4 *pf = (float4 *)(base + at[6]);
  int64_t *cell = (int64_t *)(base + at[7]), *cnt = (int64_t *)(base + at[8]);
  R.rowptr = (int64_t *)(base + at[9]);
  double *box = (double *)(base + at[10]);
  int *err = (int *)(base + at[11]);
  void *tmp = base + at[12];
  int64_t *cells = nullptr;  // first and last node of each cell
  auto done = [&](cudaError_t r) {
    cudaFree(cells);
    return r;
  };
#define NS_TRY(call)                                  \
  do {                                                \
    if ((e = (call)) != cudaSuccess) return done(e);  \
  } while (0)
  NS_TRY(cudaMemcpyAsync(dx, x, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, s));
  k_bbox<<<kBoxBlocks, 256, 0, s>>>(n, dx, box);
  std::vector<double> hb(8 * kBoxBlocks);
  NS_TRY(cudaMemcpyAsync(hb.data(), box, sizeof(double) * hb.size(), cudaMemcpyDeviceToHost, s));
  NS_TRY(cudaStreamSynchronize(s));
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  for (int b = 0; b < kBoxBlocks; b++) {
    if (hb[8 * b + 6] != 0.) {
      why = "non-finite coordinate";
      return done(cudaErrorInvalidValue);
    }
    for (int d = 0; d < 3; d++) {
      lo[d] = std::min(lo[d], hb[8 * b + d]);
      hi[d] = std::max(hi[d], hb[8 * b + 3 + d]);
    }
  }
  const Grid g = grid_of(lo, hi, horizon);
  const NearBand band = near_band(g);
  const int64_t ncell = g.nc[0] * g.nc[1] * g.nc[2];
  NS_TRY(cudaMalloc(&cells, sizeof(int64_t) * 2 * ncell));
  NS_TRY(cudaMemsetAsync(cells, 0, sizeof(int64_t) * 2 * ncell, s));
  NS_TRY(cudaMemsetAsync(err, 0, sizeof(int), s));
  NS_TRY(cudaMemsetAsync(cnt + n, 0, sizeof(int64_t), s));
  k_cell_keys<<<blocks(n, 256), 256, 0, s>>>(n, dx, g, nullptr, keys, vals);
  NS_TRY(cub::DeviceRadixSort::SortPairs(tmp, sort_b, keys, keys2, vals, perm, (int)n, 0, 64, s));
  k_gather_sorted<<<blocks(n, 256), 256, 0, s>>>(n, 4, dx, perm, g, pos, pf, cell);
  k_cell_ranges<<<blocks(n, 256), 256, 0, s>>>(n, cell, cells, cells + ncell);
  k_neighbors<false, true><<<blocks(n, 128), 128, 0, s>>>(n, 4, pos, pf, band, cell, g, cells,
                                                          cells + ncell, perm, cnt, nullptr,
                                                          nullptr, err);
  NS_TRY(cudaGetLastError());
  NS_TRY(cub::DeviceScan::ExclusiveSum(tmp, scan_b, cnt, R.rowptr, n + 1, s));
  int herr = 0;
  NS_TRY(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
  NS_TRY(cudaMemcpyAsync(&R.nnz, R.rowptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  NS_TRY(cudaStreamSynchronize(s));
  if (herr == DEVERR_ROW_TOO_LONG) {
    why = "a neighbour row exceeds the supported maximum";
    return done(cudaErrorInvalidValue);
  }
  if (want_cols) {
    NS_TRY(cudaMalloc(&R.cols, sizeof(int) * (R.nnz + 1)));
    k_neighbors<true, true><<<blocks(n, 128), 128, 0, s>>>(n, 4, pos, pf, band, cell, g, cells,
                                                           cells + ncell, perm, nullptr, R.rowptr,
                                                           R.cols, err);
    k_sort_rows<false><<<blocks(n, 4), 128, 0, s>>>(n, R.rowptr, perm, R.cols);
    NS_TRY(cudaGetLastError());
  }
#undef NS_TRY
  return done(cudaSuccess);
}

}  // namespace nlm
