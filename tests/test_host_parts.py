"""Parts of the kernels that are compiled for the host too, on the host."""
import os
import subprocess

import pytest

from ppc_b200 import build


def _run(tmp_path, code, *flags):
    """Compiles a program over the library's headers and returns what it prints."""
    src, exe = tmp_path / "t.cpp", str(tmp_path / "t")
    src.write_text(code)
    subprocess.run([build.CXX, "-std=c++17", "-O1", "-ffp-contract=off", "-I" + build.SRC,
                    "-I" + os.path.join(build.CUDA_HOME, "include"), *flags, str(src), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
    return r.stdout


def test_step_totals_beyond_32_bits(tmp_path):
    out = _run(tmp_path, """
#include <cstdio>
#include "propagate.cuh"
int main() {
  ppcb::StepTotal t{0};
  for (int k = 0; k < 5; k++) t.add(4000000000u);
  printf("%llu", (unsigned long long)t.n);
}
""")
    assert int(out) == 5 * 4000000000


def test_cell_index_of_the_kernel_does_not_overflow(tmp_path):
    """The kernel's branch of sg_cell, with the intrinsics that it uses defined here, over grids
    up to the largest: the cell's row and column, without signed overflow on the way."""
    out = _run(tmp_path, """
#include <cmath>
#include <cstdio>
#include <cstring>
#include <cstdint>
#define __CUDA_ARCH__ 1000
static float __saturatef(float x) { return x > 0 ? (x < 1 ? x : 1.f) : 0.f; }
static int __float_as_int(float x) { int i; std::memcpy(&i, &x, 4); return i; }
static uint32_t __float_as_uint(float x) { uint32_t i; std::memcpy(&i, &x, 4); return i; }
static float __uint_as_float(uint32_t i) { float x; std::memcpy(&x, &i, 4); return x; }
using std::fmaf;
#include "strgrid.h"
int main() {
  const int sizes[][2] = {{2, 2}, {2, 8192}, {3, 5}, {127, 129}, {128, 128}, {8192, 2}};
  long bad = 0, n = 0;
  for (auto& z : sizes) {
    ppcb::StrGridParams g;  // cells of a metre, the first one centred on the origin
    g.nx = z[0]; g.ny = z[1]; g.cu = g.nx - 1; g.cv = g.ny - 1; g.su = 1 / g.cu; g.sv = 1 / g.cv; g.ou = g.ov = 0;
    g.on = 1;
    g.base = (int32_t)(0u - (uint32_t)ppcb::kSgMagicBits * (uint32_t)(g.nx + 1));
    for (int j = -1; j <= g.ny; j++)
      for (int i = -1; i <= g.nx; i++, n++) {
        const int ci = i < 0 ? 0 : i < g.nx ? i : g.nx - 1, cj = j < 0 ? 0 : j < g.ny ? j : g.ny - 1;
        bad += ppcb::sg_cell(g, i + 0.2f, j - 0.2f) != cj * g.nx + ci;
      }
    bad += ppcb::sg_cell(g, NAN, NAN) != 0;
  }
  printf("%ld %ld", bad, n);
}
""", "-fsanitize=signed-integer-overflow", "-fsanitize-undefined-trap-on-error")
    bad, n = map(int, out.split())
    assert bad == 0 and n > 60_000


@pytest.mark.parametrize("reach,spacing", [("2000", "uni(0, 2.5)"), ("std::pow(10., uni(1, 6))", "uni(-1, 2.5)")],
                         ids=["detector", "far"])
def test_tilt_cells_give_the_interval_of_the_search(tmp_path, reach, spacing):
    """The 1-d tilt interval from the cells (the kernel's expressions, on the host) against the
    search among the radii: on the radii and a few ulps from them, on the cells' edges, far outside,
    for infinities and NaN.  Maps of 2 to 79 radii from up to `reach` m, 10^spacing m apart."""
    out = _run(tmp_path, """
#include <cstdio>
#include <random>
#include "tilt.h"
using namespace ppcb;
int main() {
  std::mt19937 g(5);
  auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(g); };
  long bad = 0, points = 0, maps = 0, refused = 0;
  for (int m = 0; m < 4000; m++) {
    const int lnum = m % 4 == 0 ? 2 : m % 4 == 1 ? 3 : std::uniform_int_distribution<int>(4, 79)(g);
    float lr[PPCB_LMAX] = {0};
    lr[0] = (float)(uni(-1, 1) * REACH);
    const double step = std::pow(10., SPACING);
    for (int k = 1; k < lnum; k++) lr[k] = (float)(lr[k - 1] + step * uni(0.9, 1.1));
    TiltFast f{};
    float2 cells[kTiltCells];
    if (!tilt_cells(lr, lnum, f, cells)) {
      refused++;
      continue;
    }
    maps++;
    auto check = [&](float nr) {
      points++;
      bad += tilt_cell_interval(f, cells, nr) != tilt_interval(lnum, [&](int i) { return lr[i]; }, nr);
    };
    for (float x : {INFINITY, -INFINITY, NAN, 1e30f, -1e30f, 3e38f, -3e38f, 0.f}) check(x);
    for (int k = 0; k < lnum; k++) {
      float a = lr[k], b = lr[k];
      for (int i = 0; i < 8; i++) {
        check(a), check(b);
        a = std::nextafterf(a, INFINITY), b = std::nextafterf(b, -INFINITY);
      }
    }
    for (int c = -2; c < 2 * kTiltCells + 2; c++) {  // the cells' edges and centres
      const float x = (float)((f.off - c / (2.0 * (kTiltCells - 1))) / -f.scale);
      check(x), check(std::nextafterf(x, INFINITY)), check(std::nextafterf(x, -INFINITY));
    }
    for (int i = 0; i < 300; i++) check((float)uni(lr[0] - step, lr[lnum - 1] + step));
  }
  printf("%ld %ld %ld %ld", bad, points, maps, refused);
}
""", "-DREACH=" + reach, "-DSPACING=" + spacing)
    bad, points, maps, refused = map(int, out.split())
    assert bad == 0 and maps > 2000 and points > 1_000_000 and refused > 0, out
