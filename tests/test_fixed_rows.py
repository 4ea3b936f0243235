"""The batched path's Bessel rows for a shell close to an ECP centre (z below the
range of test_fixed.py), on the host against 128-bit floats.

Bars.  In the first table interval (z < 1/200) the rows l <= 5 are the reference's
polynomial about 0 (those above are 0 there), tabulated by octaves: the argument is
three truncated products (2^-60), which z^l magnifies by l; a Horner step is off by 2.5
units (a truncated product, a rounded coefficient) and halves the earlier ones' error,
5 units of 2^-61 of the octave's largest value, which is 2^l times its smallest: 0.7
units of 2^-53 for l = 5, and the rounding to double adds half an ulp: 1.75 units of
2^-53 relative to the polynomial itself.  Beyond it, relative to
the row at the nearest table point: no larger than the polynomial about that point in
doubles at the rounded argument."""
import os
import subprocess

import pytest

from tests.helpers import ROOT

SRC = r"""
#include "ecp_tables.cpp"
#include "ecp_fixed.h"
#include <cstdio>
#include <quadmath.h>
using namespace ecpgb;
typedef __float128 Q;
int main() {
  u64 s = 88172645463325252ull;
  auto bits = [&] { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  auto uni = [&] { return (bits() >> 11) * 0x1p-53; };
  HostTables t;
  build_tables({5, 4, 1024, 1e-12, 1e-14, {}}, t);
  const int HL1 = t.besselHL + 1;
  double zero = 0, first = 0, wf[9] = {0}, wx[9] = {0};
  for (int k = 0; k < 200000; k++) {
    const double r = 0.01 + 10 * uni(), zt = k % 2 ? std::exp(std::log(1e-30) + (std::log(0.005) - std::log(1e-30)) * uni())
                                                   : 0.005 + 0.045 * uni();
    const double sv = zt / r;
    const Q z = (Q)sv * (Q)r;
    double K[16];
    fx_bessel_rows(t.besselX.data(), t.besselXA.data(), HL1, 8, xf_mul(xf_times100(xf_from(sv)), xf_from(r)), {0, 0}, 0, K);
    if (z < (Q)0.005L - 1e-15Q) {
      for (int l = 0; l <= 8; l++) {
        const double *q = &t.besselH[(size_t)l * 6];
        Q e = 0;
        for (int j = 5; j >= 0; j--) e = e * z + q[j];
        if (l > 5) zero += K[l] != 0 || e != 0;
        else first = std::fmax(first, std::fabs((double)(((Q)K[l] - e) / e)));
      }
    } else if (z > (Q)0.005L + 1e-15Q) {
      const double zd = sv * r;
      const int i = (int)std::floor((double)(z * 100) + 0.5);
      for (int l = 0; l <= 8; l++) {
        const double *q = &t.besselH[((size_t)i * HL1 + l) * 6];
        const Q x = z - (Q)i / 100;
        Q e = 0;
        double ed = 0;
        for (int j = 5; j >= 0; j--) { e = e * x + q[j]; ed = std::fma(ed, zd - t.besselZ[i], q[j]); }
        if (e < 0) e = 0;  // (no K_l is negative; the cut series of the highest rows can be)
        if (ed < 0) ed = 0;
        wf[l] = std::fmax(wf[l], std::fabs((double)((K[l] - e) / q[0])));
        wx[l] = std::fmax(wx[l], std::fabs((double)((ed - e) / q[0])));
      }
    }
  }
  double K0[16];
  fx_bessel_rows(t.besselX.data(), t.besselXA.data(), HL1, 8, {0, 0}, {0, 0}, 0, K0);
  for (int l = 1; l <= 8; l++) zero += K0[l] != 0.0;
  int worse = 0;
  for (int l = 0; l <= 8; l++) worse += wf[l] > wx[l];
  std::printf("%.4g %d %g %g", first * 0x1p53, worse, K0[0], zero);
  for (int l = 0; l <= 8; l++) std::printf(" %.2f/%.2f", std::log2(wf[l]), std::log2(wx[l]));
  std::printf("\n");
}
"""


def _run(tmp_path, source):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(source)
    r = subprocess.run(["g++", "-O2", "-std=gnu++17", "-I", os.path.join(ROOT, "libecp_gb300", "csrc"), "-I",
                        os.path.join(ROOT, "include"), src, "-lquadmath", "-o", exe], capture_output=True, text=True)
    if r.returncode and "quadmath" in r.stderr:
        pytest.skip("no libquadmath on this machine")
    assert r.returncode == 0, r.stderr
    return subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()


def test_rows_near_a_centre_are_as_precise_as_doubles(tmp_path):
    o = _run(tmp_path, SRC)
    print(o)
    assert float(o[0]) <= 1.75 and int(o[1]) == 0 and float(o[2]) == 1.0 and float(o[3]) == 0.0, o
