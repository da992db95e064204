"""The float-pair exponential (csrc/ff32.cuh) against extended precision, on the host.

Its argument is reduced by n ln 2 (n up to 43 here: 43 ln 2 2^-49 = 5e-14) and seven
products and sums of pairs, 2^-44 each at most, give the result: 4e-13 in all. With the
terms from r^5 on in FP32 alone it was 2.5e-12."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caracal_gb300", "csrc")

DRIVER = r"""
#define __device__
#define __host__
#define __forceinline__ inline
#include <cmath>
#include <cstring>
#include <math.h>
static inline float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static inline unsigned __float_as_uint(float f) { unsigned u; std::memcpy(&u, &f, 4); return u; }
static inline int __double2hiint(double x) { long long u; std::memcpy(&u, &x, 8); return (int)(u >> 32); }
static inline int __double2loint(double x) { long long u; std::memcpy(&u, &x, 8); return (int)u; }
static inline double __hiloint2double(int h, int l) {
  unsigned long long u = (unsigned long long)(unsigned)h << 32 | (unsigned)l; double x; std::memcpy(&x, &u, 8); return x;
}
#include "ff32.cuh"
#include <cstdio>
int main() {
  long double worst = 0;
  for (int i = 0; i <= 400000; ++i) {
    const double x = -30.0 + 35.0 * i / 400000.0;
    const cr::ff a{(float)x, (float)(x - (double)(float)x)};
    const cr::ff e = cr::ff_exp(a);
    const long double want = std::exp((long double)a.hi + (long double)a.lo);
    const long double d = std::fabs(((long double)e.hi + (long double)e.lo) / want - 1.0L);
    if (d > worst) worst = d;
  }
  std::printf("%.3Le\n", worst);
}
"""


def test_pair_exponential(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(DRIVER)
    (tmp_path / "cuda_runtime.h").write_text("")
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off", "-I", str(tmp_path), "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    worst = float(subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout)
    print("largest relative error", worst)
    assert worst <= 4e-13
