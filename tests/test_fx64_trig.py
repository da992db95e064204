"""Sine, cosine, erf, arc sine and large powers on the integer pipe
(csrc/fx64.cuh) against extended precision, on the host.

Sine, cosine and erf are good to an absolute 2^-58 before the rounding (half an
ulp of 1 is 2^-54), the reduction by the 64-bit 2 / pi adds |x| 2^-65: bounds
0.54 and, up to |x| = 1000, 1 in units of 2^-53.  Arc sine: one rounding plus 0.1
ulp.  x^y for 2 <= |y| < 16: the logarithm's 57 bits times y, 2.5 units."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caracal_gb300", "csrc")

DRIVER = r"""
#include "fx64.cuh"
#include <algorithm>
#include <cstdio>
#include <random>
using namespace cr;
static std::mt19937_64 gen(11);
static double unit() { return std::uniform_real_distribution<double>(0, 1)(gen); }
// rel: in units of 2^-53 of the value, else of 1
template <class F, class R>
void check(const char* name, double bound, F f, R ref, double lo, double hi, bool rel) {
  double worst = 0, at = 0;
  for (int i = 0; i < 300000; ++i) {
    double x = lo + unit() * (hi - lo);
    if (i == 0) x = lo;
    if (i == 1) x = hi;
    if (i >= 2 && i < 200) x = std::nextafter((i - 100) * 0.78539816339744831, i & 1 ? 2e9 : -2e9);
    if (i >= 200 && i < 300) x = std::ldexp(1.0, -(i - 200));
    if (x < lo || x > hi) continue;
    const long double e = ref((long double)x);
    const double d = (double)(std::fabs((long double)f(x) - e) * 0x1p53L / (rel ? std::fabs(e) : 1.0L));
    if (!(d <= worst)) worst = d, at = x;
  }
  std::printf("%s %.17g %.4f %s\n", name, at, worst, worst <= bound ? "ok" : "BAD");
}
static bool same(double a, double b) { return a == b || (a != a && b != b) || std::fabs(a - b) < 1e-16; }
int main() {
  auto S = [](double x) { double s, c; fx::sincos(x, s, c); return s; };
  auto C = [](double x) { double s, c; fx::sincos(x, s, c); return c; };
  auto sl = [](long double x) { return std::sin(x); };
  auto cl = [](long double x) { return std::cos(x); };
  check("sin", 0.54, S, sl, -8, 8, false);
  check("cos", 0.54, C, cl, -8, 8, false);
  check("sin1000", 1, S, sl, -1000, 1000, false);
  check("cos1000", 1, C, cl, -1000, 1000, false);
  check("erf", 0.54, [](double x) { return fx::erf(x); }, [](long double x) { return std::erf(x); }, -7, 7, false);
  check("asin", 1.2, [](double x) { return fx::asin(x); }, [](long double x) { return std::asin(x); }, -0.5, 0.5, true);
  check("asin0", 1.2, [](double x) { return fx::asin(x); }, [](long double x) { return std::asin(x); }, 1e-30, 1e-3, true);
  for (double y : {2.0, 7.3, 15.9, -8.0, -12.5})
    check("pow", 2.5, [y](double x) { return fx::pow(x, y); }, [y](long double x) { return std::pow(x, (long double)y); }, 0.5, 2.2, true);
  bool ok = true;
  for (double x : {0.0, -0.0, (double)INFINITY, -(double)INFINITY, (double)NAN, 5e-324, 1e-310, 1e300, -1e5, 1024.0, 6.0, -6.5, 1.1}) {
    ok &= same(S(x), std::sin(x)) && same(C(x), std::cos(x)) && same(fx::erf(x), std::erf(x)) && same(fx::asin(x), std::asin(x));
    ok &= same(fx::pow(x, 16.0), std::pow(x, 16.0)) || x == 1.1;
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
    assert out.count("\n") == 13 and "BAD" not in out
