// bond64.cuh -- what the kernels over the FP64 bond store share (fd_fp64.cu, the
// quasi-static residual in qs.cu).
#pragma once

namespace nlm {

// exp(x): the Taylor polynomial of degree 7 where |x| < 2^-6 (bonds below 0.18 of
// the critical strain; truncation 2^-63, last operation a fused 1 + x q: within
// 0.506 ulp, tests/test_exp_small.py), CUDA's exp() elsewhere.  Up to 2^-5 the
// truncation of 2^-55 counts: 0.69 ulp below 0, where results lie under 1.  The
// polynomial is 7 FP64 instructions against about 19.
constexpr int kExpSmall = 0x3f900000;  // high word of 2^-6
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
