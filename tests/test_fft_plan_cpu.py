"""The plans of the register-blocked transforms (csrc/fft.cuh), made on the host: every length up to 2^16 and some beyond that
the kernels do not take, with the array bounds checked (the plan holds a fixed number of stages), the factors' product, and
the multiplication that stands for the division by the product of the earlier factors."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "soerenpragya3dglasma_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "fft.cuh"
using namespace glasma::fft;
int main() {
  for (int n = 1; n < (1 << 16); n++) {
    int m = n;
    for (int p : {2, 3, 5})
      while (m % p == 0) m /= p;
    Plan p;
    if (make_plan(n, p) != (n > 1 && m == 1)) return std::printf("accepted %d\n", n), 1;
    if (n == 1 || m != 1) continue;
    long long product = 1;
    for (int s = 0; s < p.nstages; s++) {
      for (unsigned j = 0; product > 1 && j < 65536; j += 1 + j / 64)
        if ((unsigned)(((unsigned long long)j * p.magic[s]) >> 32) != j / (unsigned)product) return std::printf("magic %d\n", n), 2;
      product *= p.radix[s];
    }
    if (product != n) return std::printf("product %d\n", n), 3;
  }
  // 3^13, 3^19, 5^12, 2^16, 2^30, 3^10 7, 2 3^18
  for (int n : {1594323, 1162261467, 244140625, 65536, 1 << 30, 413343, 774840978}) {
    Plan p;
    if (make_plan(n, p)) return std::printf("accepted %d\n", n), 4;
  }
  return 0;
}
"""


def test_fft_plans(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "plan.cu", tmp_path / "plan"
    src.write_text(PROGRAM)
    # an index out of an array's bounds ends the program
    bounds = "-fsanitize=bounds,-fsanitize-undefined-trap-on-error"
    subprocess.run([nvcc, "-std=c++17", "-O1", "-Xcompiler", bounds, "-I", CSRC, "-o", str(exe), str(src)], check=True,
                   capture_output=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout)
