"""Parts of the kernels that are compiled for the host too, on the host."""
import os
import subprocess

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
