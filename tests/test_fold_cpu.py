"""The coordinate fold of float64 coordinates (common.cuh fold_f64) against x87
long double, bit for bit, on the host: the header's function compiled by nvcc for
the CPU.  Inputs where the pair-of-doubles form and the 128-bit integer form meet:
cell and half-cell edges and their neighbours, tiny and zero positions, positions
just below the period, and random ones."""
import platform
import shutil
import subprocess

import pytest

from ducc_b200 import build

NVCC = build.NVCC if shutil.which(build.NVCC) else shutil.which("nvcc")
SRC = r"""
#include "common.cuh"
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
using namespace dnufft;
static void x87(double x, double cf, int n, double shift, int maxi0, int &i0, double &frac) {
  volatile double tmp = x * cf;
  volatile double f = tmp - std::floor(tmp);
  volatile long double tmp2 = (long double)f * (long double)n;
  volatile long double t = tmp2 + (long double)shift;
  i0 = std::min(int(t) - n, maxi0);
  volatile long double d = tmp2 - (long double)i0;
  frac = double(d);
}
int main() {
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> u(-1, 1);
  long bad = 0;
  for (int W = 4; W <= 16; ++W)
    for (int n : {16, 18, 100, 2880, 65536, 1 << 20, (1 << 29) + 2})
      for (double cf : {1 / (2 * M_PI), 1.0, 1 / 3.7e-5})
        for (int it = 0; it < 4000; ++it) {
          const double shift = W * (-0.5) + 1 + double(n), p = 1 / cf;
          const int maxi0 = n + (W + 1) / 2 - W;
          double x = u(g) * p;
          switch (it % 8) {
            case 0: x = u(g) * p * 100; break;
            case 1: x = p * std::ldexp(u(g), -int(g() % 60)); break;
            case 2: x = p * (double(g() % (2 * (unsigned long)n)) / (2. * n)); break;
            case 3:
              x = p * (double(g() % (2 * (unsigned long)n)) / (2. * n));
              for (int j = int(g() % 3); j >= 0; --j) x = std::nextafter(x, (g() & 1) ? 1e300 : -1e300);
              break;
            case 4: x = (g() & 1) ? 0. : -std::ldexp(1., -int(g() % 300)); break;
            case 5: x = p * (1 - std::ldexp(1., -int(g() % 54))); break;
            default: break;
          }
          int i1, i2;
          double f1, f2;
          x87(x, cf, n, shift, maxi0, i1, f1);
          fold_f64(x, cf, n, shift, maxi0, i2, f2);
          if (i1 != i2 || f1 != f2) ++bad;
        }
  std::printf("%ld\n", bad);
  return bad != 0;
}
"""


@pytest.mark.skipif(NVCC is None or platform.machine() != "x86_64",
                    reason="needs nvcc and x87 long double")
def test_fold_f64_matches_long_double(tmp_path):
    src, exe = tmp_path / "fold.cu", tmp_path / "fold"
    src.write_text(SRC)
    subprocess.run([NVCC, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-I" + build.CSRC,
                    "-o", str(exe), str(src)] + build.ARCH, check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout


RANGE = r"""
#include "common.cuh"
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>
using namespace dnufft;
template <typename Tc> static long bad_cells(std::mt19937_64 &g) {
  std::uniform_real_distribution<double> u(-1, 1);
  const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
  long bad = 0;
  for (int W = 4; W <= 16; ++W)
    for (int n : {2 * ((W + 1) / 2), 16, 18, 6000, 65536, (1 << 29) + 2})
      for (double cf : {1 / (2 * M_PI), 1.0, 1 / 3.7e-5, 1e30})
        for (int it = 0; it < 200; ++it) {
          const int nsafe = (W + 1) / 2;
          if (n < 2 * nsafe) continue;
          const double shift = W * (-0.5) + 1 + double(n);
          Tc x = Tc(u(g) / cf);
          switch (it % 8) {
            case 0: x = Tc(nan); break;
            case 1: x = Tc(it & 8 ? inf : -inf); break;
            case 2: x = Tc(std::ldexp(u(g), int(g() % 2000) - 1000)); break;
            case 3: x = Tc(-std::ldexp(1., -int(g() % 1000))); break;
            case 4: x = Tc(std::ldexp(u(g), int(g() % 126))); break;
            default: break;
          }
          int i0 = 1 << 30;
          double frac = 0;
          fold<Tc>(x, cf, n, shift, n + nsafe - W, i0, frac);
          const bool finite = std::isfinite(double(x) * cf);
          if (i0 < -nsafe || i0 > n + 1 - nsafe || std::isfinite(frac) != finite) ++bad;
        }
  return bad;
}
int main() {
  std::mt19937_64 g(2);
  const long b = bad_cells<float>(g) + bad_cells<double>(g);
  std::printf("%ld\n", b);
  return b != 0;
}
"""


@pytest.mark.skipif(NVCC is None, reason="needs nvcc")
def test_fold_stays_on_the_grid_for_every_coordinate(tmp_path):
    """The first footprint cell lies in [-nsafe, n + 1 - nsafe] for coordinates
    that are not finite too (tile keys and the cells that kernels touch rest on
    it), and their weights' argument is not a number."""
    src, exe = tmp_path / "range.cu", tmp_path / "range"
    src.write_text(RANGE)
    subprocess.run([NVCC, "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-I" + build.CSRC,
                    "-o", str(exe), str(src)] + build.ARCH, check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout
