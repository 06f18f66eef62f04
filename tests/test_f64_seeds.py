"""Integer FP64 quotients and roots (csrc/e2d_f64_intdiv.h) over every FP32 seed:
each leading 24 bits of a divisor and of a radicand (both parities of its
exponent), low bits all zeros and all ones, bit for bit the IEEE operations."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "euler2d_kokkos_gb300", "csrc")

DRIVER = r"""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include "e2d_f64_intdiv.h"
using namespace e2d::f64i;
int main() {
  long bad = 0, refused = 0;
  double worst = 0.0;
  for (uint32_t k = 0; k < 1u << 23; ++k)
    for (uint32_t ones : {0u, 1u}) {
      const uint32_t hi = k >> 3, lo = (k & 7u) << 29 | (ones ? 0x1fffffffu : 0u);
      const double b = make(0x3ff00000u | hi, lo);
      const Divisor d = divisor(b);
      const double gap = 1.0 - (double)d.y * b / 4294967296.0;  // y <= 2^32 / b, short of it by less than 2^-28.6
      bad += gap < 0.0;
      worst = gap > worst ? gap : worst;
      for (double a : {1.0, make(0x3fffffffu, 0xffffffffu), make(0x3fefffffu, 0xffffffffu)}) {
        bool ok;
        const double q = quotient(a, d, ok);
        bad += q != a / b;
        refused += !ok;
      }
      for (double x : {b, 2.0 * b}) {
        bool ok;
        const double s = root(x, ok);
        bad += s != std::sqrt(x);
        refused += !ok;
      }
    }
  std::printf("%ld %ld %d\n", bad, refused, worst < std::exp2(-28.6) ? 1 : 0);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("shift", [-2, 0, 2])
def test_every_host_seed_moved_by_units_of_its_last_place(tmp_path, shift):
    src, exe = tmp_path / "driver.cpp", str(tmp_path / "driver")
    src.write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-DE2D_SEED_SHIFT={shift}", "-I" + CSRC,
                    str(src), "-o", exe], check=True)
    bad, refused, short = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    assert bad == 0 and refused == 0 and short == 1


def _leading(parity, ones):
    """Every double in [1, 2) (parity 1: [2, 4)) of these low 29 bits."""
    k = np.arange(1 << 23, dtype=np.uint64) << np.uint64(29)
    low = np.uint64((1 << 29) - 1 if ones else 0)
    return (k | low | np.uint64((1023 + parity) << 52)).view(np.float64)


@pytest.mark.gpu
@pytest.mark.parametrize("ones", [False, True])
def test_every_device_seed_of_a_quotient(gpu_lib, ones):
    """u = mx / rho and v = my / rho of the device's primitives, numerators 1
    and the double below 2."""
    import euler2d_kokkos_gb300 as e2d

    p = e2d.make_params(8, 8, gamma0=1.4)
    top = np.nextafter(2.0, 0.0)
    for rho in np.split(_leading(0, ones), 4):
        rows = np.stack([rho, np.full_like(rho, 10.0), np.ones_like(rho), np.full_like(rho, top)], 1)
        out = e2d.eval_device(p, "primitives", rows)
        assert np.array_equal(out[:, 2], 1.0 / rho) and np.array_equal(out[:, 3], top / rho)


@pytest.mark.gpu
@pytest.mark.parametrize("ones", [False, True])
@pytest.mark.parametrize("parity", [0, 1])
def test_every_device_seed_of_a_root(gpu_lib, parity, ones):
    """c = sqrt(gamma p / rho) for gamma = 2, rho = 1, at rest: p = E, c = sqrt(2 E)."""
    import euler2d_kokkos_gb300 as e2d

    p = e2d.make_params(8, 8, gamma0=2.0)
    for x in np.split(_leading(parity, ones), 4):
        rows = np.zeros((x.size, 4))
        rows[:, 0], rows[:, 1] = 1.0, 0.5 * x
        out = e2d.eval_device(p, "primitives", rows)
        assert np.array_equal(out[:, 4], np.sqrt(x))
