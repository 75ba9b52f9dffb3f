"""sqrt_refine (csrc/fmc_common.h), the root of the pair loops, compiled for the host: from estimates of
1/sqrt(x) as far off as the hardware's (20 bits) it is within an ulp of the correctly rounded root."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

SRC = r"""
#include <cstdio>
#include <random>
#include "fmc_common.h"
int main() {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> e(-40.0, 20.0), d(-1.0, 1.0);
  double worst = 0.0;
  for (int i = 0; i < 2000000; i++) {
    const double x = std::exp2(e(g)), y = (1.0 + d(g) * 0x1p-20) / std::sqrt(x), r = std::sqrt(x);
    const double ulp = std::nextafter(r, 1e300) - r;
    worst = std::fmax(worst, std::fabs(fmc::sqrt_refine(x, y) - r) / ulp);
  }
  std::printf("%.3f\n", worst);
}
"""


def test_sqrt_refine_within_an_ulp(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(PKG, "csrc"),
                    str(tmp_path / "t.cpp"), "-o", exe], check=True)
    assert float(subprocess.run([exe], check=True, capture_output=True, text=True).stdout) <= 1.0
