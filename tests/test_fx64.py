"""The integer-pipe FP64 functions (csrc/fx64.cuh) against extended precision.

The header compiles for the host with the hardware estimates replaced by FP32
values that are as inexact.  Each function is compared with the C library's
long double result over its integer path's range, at the edges of its
reductions and at arguments that leave the path.  Bounds: one rounding (0.5
ulp) plus what the fixed-point values carry, 2^-8 ulp for reciprocal, quotient
and roots (62 bits before the rounding), 0.1 for arc cosine and for exp up to
|x| = 40 (n ln 2 leaves 58 bits or more), 0.4 for exp up to 512 and for pow
(54 to 57 bits behind the integer part of the exponent)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caracal_gb300", "csrc")

DRIVER = r"""
#include "fx64.cuh"
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace cr;
static std::mt19937_64 gen(7);
static double unit() { return std::uniform_real_distribution<double>(0, 1)(gen); }
template <class F, class R>
void check(const char* name, double bound, F f, R ref, double lo, double hi, bool log_scale) {
  double worst = 0, at = 0;
  for (int i = 0; i < 300000; ++i) {
    double x = log_scale ? std::exp(std::log(lo) + unit() * (std::log(hi) - std::log(lo))) : lo + unit() * (hi - lo);
    if (i == 0) x = lo;
    if (i == 1) x = hi;
    if (i >= 2 && i < 200) x = std::nextafter(std::ldexp(1.0, i % 40 - 20), i & 1 ? 2e9 : 0.0);
    if (x < lo || x > hi) continue;
    const long double e = ref((long double)x);
    const double u = std::ldexp(1.0, std::ilogb((double)e) - 52);
    const double d = (double)(std::fabs((long double)f(x) - e) / u);
    if (!(d <= worst)) worst = d, at = x;
  }
  std::printf("%s %.17g %.4f %s\n", name, at, worst, worst <= bound ? "ok" : "BAD");
}
// equal, or neighbours (both are within one rounding of the value), or both NaN
static bool same(double a, double b) { return a == b || (a != a && b != b) || std::nextafter(a, b) == b; }
int main() {
  const double r = 0.504;
  check("rcp", r, [](double x) { return fx::rcp(x); }, [](long double x) { return 1 / x; }, 1e-300, 1e300, true);
  check("rcp1", r, [](double x) { return fx::rcp(x); }, [](long double x) { return 1 / x; }, 1.0, 2.0, false);
  check("div", r, [](double x) { return fx::div(-3.7, x); }, [](long double x) { return -3.7 / x; }, 1e-200, 1e200, true);
  check("div1", r, [](double x) { return fx::div(x, 1.7); }, [](long double x) { return x / 1.7; }, 1.0, 4.0, false);
  check("sqrt", r, [](double x) { return fx::sqrt(x); }, [](long double x) { return std::sqrt(x); }, 1e-300, 1e300, true);
  check("sqrt1", r, [](double x) { return fx::sqrt(x); }, [](long double x) { return std::sqrt(x); }, 0.9, 4.1, false);
  check("rsqrt", r, [](double x) { return fx::rsqrt(x); }, [](long double x) { return 1 / std::sqrt(x); }, 1e-300, 1e300, true);
  check("root", r, [](double x) { double a, b; fx::sqrt_rsqrt(x, a, b); return a; }, [](long double x) { return std::sqrt(x); }, 0.9, 4.1, false);
  check("iroot", r, [](double x) { double a, b; fx::sqrt_rsqrt(x, a, b); return b; }, [](long double x) { return 1 / std::sqrt(x); }, 0.9, 4.1, false);
  check("exp", 0.6, [](double x) { return fx::exp(x); }, [](long double x) { return std::exp(x); }, -40, 40, false);
  check("exp2", 0.9, [](double x) { return fx::exp(x); }, [](long double x) { return std::exp(x); }, -511, 511, false);
  check("expm", 0.9, [](double x) { return fx::exp(-x); }, [](long double x) { return std::exp(-x); }, 1e-25, 500, true);
  check("pow", 0.9, [](double x) { return fx::pow(x, -1.5309487826); }, [](long double x) { return std::pow(x, (long double)-1.5309487826); }, 0.3, 50, true);
  check("pow2", 0.9, [](double x) { return fx::pow(x, 0.4367417579); }, [](long double x) { return std::pow(x, (long double)0.4367417579); }, 1e-6, 1e6, true);
  check("acos", 0.6, [](double x) { return fx::acos(x); }, [](long double x) { return std::acos(x); }, -1, 1, false);
  check("acos0", 0.6, [](double x) { return fx::acos(x); }, [](long double x) { return std::acos(x); }, 1e-30, 0.5, true);
  check("acos1", 0.6, [](double x) { return fx::acos(1 - x); }, [](long double x) { return std::acos((long double)(1 - (double)x)); }, 1e-9, 1, true);
  const double inf = INFINITY, nan = NAN, tiny = 5e-324;
  const double xs[] = {0.0, -0.0, inf, -inf, nan, tiny, 1e-310, -1e-310, 1.7e308, -1.0, 1.0, 2.0, 0.5, 800.0, -800.0, 1e-30, 1.0 - 1e-16, 1.1};
  bool ok = true;
  for (double x : xs) {
    ok &= same(fx::rcp(x), 1 / x) && same(fx::div(1.5, x), 1.5 / x) && same(fx::div(x, 3.0), x / 3.0);
    ok &= same(fx::sqrt(x), std::sqrt(x)) && same(fx::exp(x), std::exp(x)) && same(fx::acos(x), std::acos(x));
    ok &= same(fx::pow(x, 1.5), std::pow(x, 1.5)) && same(fx::rsqrt(x), 1 / std::sqrt(x));
  }
  std::printf("edges 0 0 %s\n", ok ? "ok" : "BAD");
}
"""


def test_accuracy_and_edges(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src = tmp_path / "fx.cpp"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(tmp_path / "fx")], check=True)
    out = subprocess.run([str(tmp_path / "fx")], check=True, capture_output=True, text=True).stdout
    print(out)
    assert out.count("\n") == 18 and "BAD" not in out
