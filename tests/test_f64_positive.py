"""The sign test behind the density flag (csrc/e2d_f64_intdiv.h) against x > 0.0,
on the host build of the header."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "euler2d_kokkos_gb300", "csrc")

DRIVER = r"""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include "e2d_f64_intdiv.h"
int main() {
  int bad = 0, n = 0;
  for (double x : {0.0, 5e-324, 1e-310, 2.3e-308, 1e-10, 1.0, 1.7e308, (double)INFINITY, (double)NAN,
                   e2d::f64i::make(0x7ff00000u, 1u), e2d::f64i::make(0x7fffffffu, 0xffffffffu)})
    for (double y : {x, -x, std::copysign(x, -1.0)}) {
      bad += e2d::f64i::positive(y) != (y > 0.0);
      ++n;
    }
  std::printf("%d %d\n", bad, n);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_positive_is_greater_than_zero(tmp_path):
    src, exe = tmp_path / "driver.cpp", str(tmp_path / "driver")
    src.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, str(src), "-o", exe], check=True)
    bad, n = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    assert bad == 0 and n == 33
