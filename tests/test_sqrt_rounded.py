"""sqrt_rounded (csrc/fmc_common.h), the root of the plain path's pairs, compiled for the host: from estimates of
1/sqrt(x) as far off as the hardware's (20 bits) it is sqrt(x) correctly rounded, also where that lies closest to the
middle between two numbers (x = 1 + o ulp, o odd and small, and its multiples by 4)."""
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
  long long wrong = 0;
  auto test = [&](double x) {
    const double r = std::sqrt(x);
    for (int k = 0; k < 4; k++) wrong += fmc::sqrt_rounded(x, (1.0 + d(g) * 0x1p-20) / r) != r;
  };
  for (int i = 0; i < 2000000; i++) test(std::exp2(e(g)));
  for (int i = 0; i < 20000; i++) {
    const double x = 1.0 + i * 0x1p-52, y = 1.0 - i * 0x1p-53, z = 2.0 - i * 0x1p-52;
    for (int k = -20; k <= 10; k += 2)
      for (double v : {x, y, z, 2.0 * x, 2.0 * y}) test(std::ldexp(v, k));
  }
  std::printf("%lld\n", wrong);
}
"""


def test_sqrt_rounded_is_sqrt(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(PKG, "csrc"),
                    str(tmp_path / "t.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.strip() == "0"
