"""Integer-pipe FP64 division, square root and product (csrc/e2d_f64_intdiv.h):
bit for bit the IEEE operations, on the host build of the header (CPU) and through the
device's primitives block (GPU)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "euler2d_kokkos_gb300", "csrc")

DRIVER = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "e2d_f64_intdiv.h"
using namespace e2d::f64i;
static std::mt19937_64 r(20240607);
static double draw(int spread) {  // significands with runs of zeros and ones at either end, exponents within +-spread
  uint64_t m = r();
  switch (r() % 6) {
    case 0: m &= ~0ull << (r() % 53); break;
    case 1: m |= ~(~0ull << (r() % 53)); break;
    case 2: m = ~0ull - r() % 5; break;
    case 3: m = r() % 5; break;
    default: break;
  }
  const uint64_t e = spread ? 1023 - spread + r() % (2 * spread + 1) : 1023;
  const uint64_t b = (r() & (1ull << 63)) | (e << 52) | (m & ((1ull << 52) - 1));
  double d;
  std::memcpy(&d, &b, 8);
  return d;
}
int main() {
  long bad = 0, refused = 0, n = 0;
  for (long i = 0; i < 3000000; ++i) {
    const int spread = (i % 3 == 0) ? 0 : (i % 3 == 1) ? 40 : 490;
    const double a = (i % 64 == 0) ? std::copysign(0.0, draw(0)) : draw(spread), b = draw(spread);
    bool ok;
    const double q = quotient(a, divisor(b), ok), t = a / b;
    refused += !ok;
    bad += ok && bits(q) != bits(t);
    const double x = std::fabs(a), y = b * b;
    const double pr = product(a, b, ok);
    refused += !ok;
    bad += ok && bits(pr) != bits(a * b);
    for (double z : {x, y, std::nextafter(y, 0.0), std::nextafter(y, 1e300)}) {
      const double s = root(z, ok);
      bad += ok && bits(s) != bits(std::sqrt(z));
      ++n;
    }
  }
  // outside the range the routine says so
  bool ok = true, any = false;
  for (double d : {0.0, 1e-310, 1e300, (double)INFINITY, (double)NAN}) quotient(1.0, divisor(d), ok), any |= ok;
  for (double a : {1e-310, (double)INFINITY, (double)NAN}) quotient(a, divisor(1.5), ok), any |= ok;
  quotient(1e300, divisor(1e-140), ok), any |= ok;
  quotient(1e-300, divisor(1e140), ok), any |= ok;
  product(1e-200, 1e-200, ok), any |= ok;
  product(1e200, -1e200, ok), any |= ok;
  product(1e-310, 1.5, ok), any |= ok;
  product(0.0, (double)INFINITY, ok), any |= ok;
  product(1.0, (double)NAN, ok), any |= ok;
  for (double x : {0.0, -1.0, -0.0, 1e-310, 1e300, (double)INFINITY, (double)NAN}) root(x, ok), any |= ok;
  std::printf("%ld %ld %d\n", bad, refused, any ? 1 : 0);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_host_build_equals_ieee(tmp_path):
    src = tmp_path / "driver.cpp"
    src.write_text(DRIVER)
    exe = str(tmp_path / "driver")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(src), "-o", exe], check=True)
    bad, refused, outside = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    assert bad == 0
    assert refused == 0  # every operand of these exponents is in range
    assert outside == 0


def _doubles(rng, n, spread):
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    kind = rng.integers(0, 5, n)
    k = rng.integers(0, 53, n).astype(np.uint64)
    ones = np.uint64((1 << 52) - 1)
    m = np.where(kind == 0, m & (ones << k) & ones, m)
    m = np.where(kind == 1, m | (ones >> k), m)
    m = np.where(kind == 2, ones - (m & np.uint64(3)), m)
    m = np.where(kind == 3, m & np.uint64(3), m)
    e = (1023 + rng.integers(-spread, spread + 1, n)).astype(np.uint64)
    return ((e << np.uint64(52)) | m).view(np.float64)


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [0, 30, 300, 520])
def test_device_primitives_divide_as_ieee(gpu_lib, spread):
    """u = mx / d, v = my / d and c = sqrt(gamma p / d) of the device's
    primitives against numpy's, operands inside the integer forms' range
    (spread <= 300) and beyond it (520: the fall-back)."""
    import euler2d_kokkos_gb300 as e2d

    rng = np.random.default_rng(spread + 1)
    n = 1 << 18
    p = e2d.make_params(8, 8, smallr=1e-10, float_params=False)
    p.smallr = 1e-200
    rho = np.maximum(_doubles(rng, n, spread), 1e-200)
    mx = _doubles(rng, n, spread) * rng.choice([-1.0, 1.0, 0.0, -0.0], n)
    my = _doubles(rng, n, spread) * rng.choice([-1.0, 1.0], n)
    with np.errstate(all="ignore"):
        u, v = mx / rho, my / rho
        e = np.abs(_doubles(rng, n, min(spread, 30))) * rho + 0.5 * rho * (u * u + v * v)
        out = e2d.eval_device(p, "primitives", np.stack([rho, e, mx, my], 1))
        d, pr, c = out[:, 0], out[:, 1], out[:, 4]
        good = np.isfinite(u) & np.isfinite(v)
        want_c = np.sqrt(p.gamma0 * pr / d)
    assert np.array_equal(out[:, 2].view(np.uint64)[good], u.view(np.uint64)[good])
    assert np.array_equal(out[:, 3].view(np.uint64)[good], v.view(np.uint64)[good])
    fin = np.isfinite(want_c)
    assert fin.sum() > n // 4
    assert np.array_equal(c[fin], want_c[fin])
