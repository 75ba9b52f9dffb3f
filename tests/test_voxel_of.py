"""voxel_of (csrc/fmc_device.cuh), compiled for the host, where the drop-in and the plain calls place their sites: every
coordinate, also one that is no number or infinite, falls into a voxel of the cell."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "fmc_device.cuh"
int main() {
  const double bad[] = {0.0, 12.5, -3.0, 24.999999999999996, 25.0, 1e9, -1e9, 1e300, -1e300, INFINITY, -INFINITY, NAN};
  fmc::DevSystem S;
  std::memset(&S, 0, sizeof(S));
  S.nvox[0] = 12, S.nvox[1] = 13, S.nvox[2] = 14;
  for (int i = 0; i < 3; i++) S.cell.rh[4 * i] = 0.04;
  S.cell.slab[0] = S.cell.slab[3] = 0.04;
  S.cell.zlo = -2.0;
  S.cell.rdz = 0.5;
  int out = 0;
  for (int imcon = 1; imcon <= 7; imcon++)
    for (double x : bad)
      for (double y : bad)
        for (double z : bad) {
          S.cell.imcon = imcon;
          const int v = fmc::voxel_of(S, x, y, z);
          if (v < 0 || v >= 12 * 13 * 14) out++;
        }
  std::printf("%d\n", out);
}
"""


def test_every_position_has_a_voxel(tmp_path):
    nvcc = os.environ.get("NVCC", shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")
    if not os.path.exists(nvcc):
        pytest.skip("no CUDA compiler")
    (tmp_path / "t.cu").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([nvcc, "-O2", "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"), str(tmp_path / "t.cu"), "-o",
                    exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.strip() == "0"
