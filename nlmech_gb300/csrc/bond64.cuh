// bond64.cuh -- what the kernels over the FP64 bond store share (fd_fp64.cu, the
// quasi-static residual in qs.cu).
#pragma once

#include "common.cuh"

namespace nlm {

// exp(x): the Taylor polynomial of degree 7 where |x| < 2^-5 (bonds below a
// quarter of the critical strain; truncation 2^-55, last operation a fused
// 1 + x q, so within 0.53 ulp), CUDA's exp() elsewhere.  The polynomial is 7
// FP64 instructions against about 19.
constexpr int kExpSmall = 0x3fa00000;  // high word of 2^-5
__device__ __forceinline__ double exp_small(double x) {
  double q = 1. / 5040.;
  q = __fma_rn(q, x, 1. / 720.);
  q = __fma_rn(q, x, 1. / 120.);
  q = __fma_rn(q, x, 1. / 24.);
  q = __fma_rn(q, x, 1. / 6.);
  q = __fma_rn(q, x, 0.5);
  q = __fma_rn(q, x, 1.);
  return __fma_rn(q, x, 1.);
}
__device__ __forceinline__ int hi_abs(double x) { return __double2hiint(x) & 0x7fffffff; }
__device__ __forceinline__ double exp64(double x) {
  return hi_abs(x) < kExpSmall ? exp_small(x) : exp(x);
}

// Break threshold words (b64_thr): bit 31 marks a bond of a no-fail node.
constexpr int kThrTough = (int)0x80000000u, kThrInf = 0x7ff00000;

}  // namespace nlm
