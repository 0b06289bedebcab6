"""exp_small (bond64.cuh), compiled for the host from the same header, against
long double over the arguments that it is used for: within 0.53 ulp, what one
rounding of a result with an error of 2^-58 leaves."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#define __device__
#define __forceinline__ inline
static double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static int __double2hiint(double x) {
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return (int)(b >> 32);
}
using std::exp;
#include "bond64.cuh"
int main() {
  double worst = 0., at = 0., top = 0.;
  for (int s = -1; s <= 1; s += 2)
    for (int e = -60; e <= 2; e++)
      for (int k = 0; k < 4000; k++) {
        const double x = s * std::ldexp(1. + (k + 0.37) / 4000., e);
        if (!(nlm::hi_abs(x) < nlm::kExpSmall)) continue;
        if (std::fabs(x) > top) top = std::fabs(x);
        const long double t = expl((long double)x);
        const double d = (double)t;
        const double ulp = d < 1. ? 0x1p-53 : 0x1p-52;
        const double err = (double)std::fabs((long double)nlm::exp_small(x) - t) / ulp;
        if (err > worst) worst = err, at = x;
      }
  std::printf("%.4f %.6g %.6g\n", worst, at, top);
}
"""


def test_error_over_its_range(tmp_path):
    src, exe = tmp_path / "e.cpp", str(tmp_path / "e")
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", str(src), "-o", exe,
                           "-I", os.path.join(ROOT, "nlmech_gb300", "csrc"),
                           "-I", os.path.join(ROOT, "include")])
    worst, at, top = map(float, subprocess.check_output([exe]).split())
    assert top > 1e-3  # the range was met
    assert worst <= 0.53, (worst, at)
