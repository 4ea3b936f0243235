"""Rounding of an integer mantissa and exponent to double at the ends of its range
(xf_to_double): infinity above the largest double, 0 below the smallest normal one."""
import os
import subprocess

from tests.helpers import ROOT

SRC = r"""
#include "ecp_fixed.h"
#include <cmath>
#include <cstdio>
using namespace ecpgb;
int main() {
  const u64 one = 1ull << 63;
  int bad = 0;
  for (int e = -1200; e <= 4000; e++) {
    const double v = xf_to_double(one, e - 63, 0), w = xf_to_double(one >> 9, e - 54, 0x80000000u);
    const double x = e < -1022 ? 0.0 : std::ldexp(1.0, e);  // infinity from 1024 on
    bad += v != x || w != -x;
  }
  bad += xf_to_double(~0ull, 1023 - 63, 0) != INFINITY;           // rounds up past the largest
  bad += xf_to_double(~0ull << 11, 1023 - 63, 0) != 0x1.fffffffffffffp1023;
  bad += xf_to_double(0, 3000, 0) != 0.0;
  std::printf("%d\n", bad);
}
"""


def test_ends_of_the_range(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-I", os.path.join(ROOT, "libecp_gb300", "csrc"), src, "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout.strip() == "0"
