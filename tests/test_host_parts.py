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
