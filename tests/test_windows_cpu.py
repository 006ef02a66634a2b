"""The cells of the register windows (spread_run.cuh, spread_run3.cuh,
interp_run.cuh, interp_run3.cuh) on the host: for every support, every accepted
length of an oversampled axis up to 64 cells (the smallest is 2 nsafe) and every
first cell, all cells of the window - also those that no finite point touches -
wrap to the grid cell they stand for."""
import shutil
import subprocess

import pytest

from ducc_b200 import build

NVCC = build.NVCC if shutil.which(build.NVCC) else shutil.which("nvcc")
SRC = r"""
#include "interp_run3.cuh"
#include <cstdio>
using namespace dnufft;
static long bad = 0;
template <int (*WRAP)(int, int) = wrap3> static void axis(int W, int lb, int width) {
  const int nsafe = (W + 1) / 2;
  for (int n = 2 * nsafe; n <= 64; n += 2)
    for (int t = 0; t <= n + 1; ++t) {
      const int start = (t >> lb << lb) - nsafe;
      if (t - nsafe + W > start + width) ++bad;      // the footprint fits the window
      for (int c = start; c < start + width; ++c)
        if (WRAP(c, n) != ((c % n) + n) % n) ++bad;
    }
}
template <int W> static void both() {
  using D2 = RunShape<double, W>;
  axis(W, 3, D2::ROWS); axis(W, 3, D2::CELLS);
  using D3 = Run3Shape<double, W>;
  axis(W, D3::LB, D3::SPAN); axis(W, D3::LB, D3::ROWS); axis(W, D3::LB, D3::CELLS);
  using I2 = InterpShape<W>;
  axis(W, 3, I2::ROWS); axis(W, 3, I2::COLS);
  using I3 = Interp3Shape<W>;
  axis(W, I3::LB, I3::SPAN); axis(W, I3::LB, I3::ROWS); axis(W, I3::LB, I3::COLS);
  if constexpr (W <= 8) {
    using F2 = RunShape<float, W>;
    axis<run_wrap<W>>(W, 3, F2::ROWS); axis<run_wrap<W>>(W, 3, F2::CELLS);
    using F3 = Run3Shape<float, W>;
    axis(W, F3::LB, F3::PLANES); axis(W, F3::LB, F3::ROWS); axis(W, F3::LB, F3::CELLS);
  }
}
int main() {
  both<4>(); both<5>(); both<6>(); both<7>(); both<8>(); both<9>(); both<10>(); both<11>();
  both<12>(); both<13>(); both<14>(); both<15>(); both<16>();
  std::printf("%ld\n", bad);
  return bad != 0;
}
"""


@pytest.mark.skipif(NVCC is None, reason="needs nvcc")
def test_window_cells_wrap_onto_the_grid(tmp_path):
    src, exe = tmp_path / "win.cu", tmp_path / "win"
    src.write_text(SRC)
    r = subprocess.run([NVCC, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I" + build.CSRC,
                        "-o", str(exe), str(src)] + build.ARCH, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout
