"""pass_stamp and slot_arrived (csrc/fmc_common.h), compiled for the host: a slot of which some words are still the
last pass's is never taken with an energy that is not the new pass's, whatever the energies: equal, zeros of both
signs, short, full, no numbers, and those that deceive a stamp which only xors its words."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

# Every mix of old and new words of one slot; prints how many were taken wrongly, and how many complete ones were not.
SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "fmc_common.h"
typedef unsigned long long word;
static word bits(double d) { word u; std::memcpy(&u, &d, 8); return u; }
static double number(word u) { double d; std::memcpy(&d, &u, 8); return d; }
static word rotr(word u, int n) { return n ? u >> n | u << (64 - n) : u; }
static long long wrong, missed;
struct Slot { double e[2], seq; };

static void mixes(const Slot& a, const Slot& b, int n) {
  for (int m = 0; m < 1 << (n + 1); m++) {
    double w[3], out[2] = {0, 0};
    for (int i = 0; i < n; i++) w[i] = (m >> i & 1 ? b : a).e[i];
    const Slot& s = m >> n & 1 ? b : a;
    w[n] = fmc::pass_stamp(s.seq, s.e[0], n > 1 ? s.e[1] : 0.0);
    const bool taken = fmc::slot_arrived(w, b.seq, n, out), whole = m == (1 << (n + 1)) - 1;
    if (whole && !taken) missed++;
    for (int i = 0; taken && i < n; i++)
      if (bits(out[i]) != bits(b.e[i])) { wrong++; break; }
  }
}

int main() {
  std::mt19937_64 g(11);
  auto energy = [&]() {
    const double special[] = {0.0, -0.0, 1.0, -1.25, INFINITY, NAN, 5e-324, -1e300};
    const int kind = g() % 4;
    const double x = std::ldexp((double)(long long)(g() % 2000001) - 1e6, (int)(g() % 40) - 30);
    return kind == 0 ? special[g() % 8] : (kind == 1 ? (double)(int)(g() % 64) / 16.0 : (kind == 2 ? (double)(float)x : x * 0.1));
  };
  for (int i = 0; i < 400000; i++) {
    Slot a, b;
    a.seq = i < 1000 ? i : (double)(g() % (1ULL << (1 + i % 50)));
    b.seq = a.seq + 1 + (i & 1 ? g() % 3 : 0);
    for (int k = 0; k < 2; k++) {
      a.e[k] = energy();
      b.e[k] = g() % 3 ? energy() : a.e[k];
    }
    if (i == 0) a.e[0] = a.e[1] = number(0);  // memory as the slots begin
    mixes(a, b, 1);
    mixes(a, b, 2);
    if (i % 100) continue;
    // the new energy that undoes the change of the stamp, wherever a stamp of xors puts it
    const word d = bits(fmc::pass_stamp(a.seq, a.e[0], a.e[1])) ^ bits(fmc::pass_stamp(b.seq, a.e[0], a.e[1]));
    for (int r = 0; r < 64; r++)
      for (int k = 0; k < 2; k++) {
        Slot c = b;
        c.e[k] = number(bits(a.e[k]) ^ rotr(d, r));
        mixes(a, c, 1);
        mixes(a, c, 2);
      }
  }
  std::printf("%lld %lld\n", wrong, missed);
}
"""


def test_no_mix_of_two_passes_is_taken(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(PKG, "csrc"), str(tmp_path / "t.cpp"), "-o", exe],
                   check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split() == ["0", "0"]
