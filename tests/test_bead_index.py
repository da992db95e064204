"""The force kernels' index of a thread's evaluation (csrc/bead_rows.cuh), on the host.

With four threads per evaluation the thread index passes 2^31 at 2^29 evaluations, an
eighth of what the int count allows.  Every thread of the blocks at the edges of the
range must find its own evaluation, and evaluations past the count must read as past it."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "caracal_gb300", "csrc")

DRIVER = r"""
#define __host__
#define __device__
#include "bead_rows.cuh"
#include <cstdio>
#include <initializer_list>
int main() {
  long long bad = 0;
  for (int L : {1, 4})
    for (long long n : {1LL, 31LL, 32LL, 33LL, 536870911LL, 536870912LL, 536870913LL, 2147483647LL}) {
      // the launch: blocks of 128 threads, 128 / L evaluations each
      const int bs = 128 / L, nb = (int)n / bs + ((int)n % bs != 0);
      for (int b : {0, nb / 2, nb - 1})
        for (unsigned t = 0; t < 128; ++t) {
          const long long want = (long long)b * bs + t / (unsigned)L;
          const size_t e = cr::evaluation_of((unsigned)b, 128, t, L);
          bad += e != (size_t)want || (e < (size_t)n) != (want < n);
        }
    }
  const cr::BeadRows r = cr::distinct_rows(32);
  bad += r.row(2147483647u) != 2147483647u / 17u * (size_t)32 + 2147483647u % 17u;
  std::printf("%lld\n", bad);
}
"""


def test_evaluation_index(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.strip() == "0"
