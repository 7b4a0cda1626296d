"""The check that a caller's device buffer lies inside its allocation (csrc/extent.h), on the host: every buffer of a few bytes
around an allocation, against the definition, and addresses at the end of the address space, where sums would wrap."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "soerenpragya3dglasma_gb300", "csrc")

PROGRAM = r"""
#include "extent.h"
using glasma::extent_holds;
int main() {
  for (unsigned size = 0; size < 6; size++)
    for (unsigned p = 90; p < 110; p++)
      for (unsigned bytes = 0; bytes < 12; bytes++)
        if (extent_holds(100, size, p, bytes) != (p >= 100 && p + bytes <= 100 + size)) return 1;
  const uintptr_t end = ~(uintptr_t)0;
  if (!extent_holds(end - 15, 16, end - 7, 8)) return 2;
  if (extent_holds(end - 15, 16, end - 7, 9)) return 3;
  if (extent_holds(end - 15, 16, end - 7, ~(size_t)0)) return 4;
  if (extent_holds(4096, 16, 4104, ~(size_t)0 - 4000)) return 5;
  return 0;
}
"""


def test_extent_holds(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    src, exe = tmp_path / "extent.cpp", tmp_path / "extent"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC, "-o", str(exe), str(src)], check=True, timeout=120)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
