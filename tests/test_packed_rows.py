"""The type-1 tables' packed Bessel rows (fx_bessel_packed), on the host: a row keeps
its own exponent, so it carries the bits of the row it was packed from -- at least a
double's 53, whatever its size against K_0.

Bar: the packed mantissa is cut to 58 bits, at most 2^-57 of the row (2^-57 exactly
where a row's leading bit is its top bit)."""
import os
import subprocess

from tests.helpers import ROOT

SRC = r"""
#include "ecp_tables.cpp"
#include "ecp_fixed.h"
#include <cstdio>
using namespace ecpgb;
int main() {
  u64 s = 88172645463325252ull;
  auto bits = [&] { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  auto uni = [&] { return (bits() >> 11) * 0x1p-53; };
  HostTables t;
  build_tables({5, 4, 1024, 1e-12, 1e-14, {}}, t);
  const int HL1 = t.besselHL + 1;
  double worst = 0;
  long clipped = 0, nonzero = 0;
  for (int k = 0; k < 400000; k++) {
    const double r = 0.01 + 10 * uni(), zt = k == 0 ? 0.0
                     : k % 3 == 0 ? std::exp(std::log(1e-30) + (std::log(0.05) - std::log(1e-30)) * uni())
                     : k % 3 == 1 ? 0.005 + 3 * uni() : 300 * uni() * uni();
    const xf z100 = xf_mul(xf_times100(xf_from(zt / r)), xf_from(r));
    xf row[16];
    fx_bessel(t.besselX.data(), t.besselXA.data(), HL1, 8, z100, [&](int l, u64 v, int scale) { row[l] = {v, -scale}; });
    u64 K[16];
    const RowBase b = fx_bessel_packed(t.besselX.data(), t.besselXA.data(), HL1, 8, z100, K);
    for (int l = 0; l <= 8; l++) {
      xf p = row_packed(K[l]);
      p.e += b.e0 - l * b.t;
      if (row[l].m == 0) { nonzero += p.m != 0; continue; }
      const xf n = xf_norm(row[l]);
      if (p.m >> 63 == 0) { clipped++; continue; }
      const double d = std::ldexp((double)(i64)(n.m - p.m), -63) + (n.e != p.e);
      worst = std::fmax(worst, std::fabs(d));
    }
  }
  std::printf("%.4f %ld %ld\n", std::log2(worst), clipped, nonzero);
}
"""


def test_packed_rows_keep_their_own_exponent(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-I", os.path.join(ROOT, "libecp_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), src, "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    print(out)
    # no row is cut for its size
    assert float(out[0]) <= -57 and int(out[1]) == 0 and int(out[2]) == 0, out
