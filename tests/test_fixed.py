"""The 64-bit integer-mantissa arithmetic of the batched path
(libecp_gb300/csrc/ecp_fixed.h), compiled for the host: the exponential, the
reciprocal, the rounding to double, and the Bessel rows over the whole
argument range against 128-bit floats.

Bars, from the operations: an exponential is a 62-bit table value times a
polynomial cut at 2^-60, three truncated 64-bit products -- below 2^-58 before
the rounding, so at most 2^-53 (1 + 2^-5) after it; a Bessel row rounds once and
its argument 100 s r is three truncated products (2^-61 of the argument), which
a row magnifies by |z K'/K| <= l + 1 + z / (2 z) -- 2 units of 2^-53 for l <= 2
where the row is not small against its table interval, and the double rows'
own error beyond."""
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
  double we = 0, wd = 0, wr = 0, wm = 0;
  int pack = 0;
  for (int k = 0; k < 400000; k++) {
    i64 E = (i64)bits();
    if (k % 2) E >>= 5;
    if (k % 3 == 0) E >>= 9;
    const xf v = fx_exp(E);
    const Q ex = expq((Q)E * ldexpq(1, -53));
    we = std::fmax(we, std::fabs((double)((ldexpq((Q)v.m, v.e) - ex) / ex)));
    if (v.e > -1000 && v.e < 950) wd = std::fmax(wd, std::fabs((double)(((Q)xf_to_double(v.m, v.e, 0) - ex) / ex)));
    const u64 x = bits() | (1ull << 63);
    wr = std::fmax(wr, std::fabs((double)((Q)fx_recip(x) * (Q)x * ldexpq(1, -126) - 1)));
    const i64 a = (i64)bits() >> (k % 40);
    const u64 b = bits() >> 1 >> (k % 7);
    wm = std::fmax(wm, std::fabs((double)((Q)mul_hi_s(a, fx_split(b)) - (Q)a * (Q)b * ldexpq(1, -64))));
    double d;
    const u64 db = bits() & 0x7fffffffffffffffull;
    std::memcpy(&d, &db, 8);
    if (d > 1e-300 && d < 1e300) {
      const xf f = xf_from(d);
      pack += xf_to_double(f.m >> 3, f.e + 3, 0x80000000u) != -d;
    }
  }
  HostTables t;
  build_tables({5, 4, 1024, 1e-12, 1e-14, {}}, t);
  const int HL1 = t.besselHL + 1, AS = HL1 < 6 ? 6 : HL1;
  double wf[9] = {0}, wx[9] = {0}, zero = 0;
  for (int k = 0; k < 100000; k++) {
    const double r = 0.1 + 10 * uni(), sv = (k % 2 ? 16 * uni() : 16 + 200 * uni() * uni()) / r;
    const Q z = (Q)sv * (Q)r;
    if (z < 0.02) continue;
    double K[16];
    fx_bessel_rows(t.besselX.data(), t.besselXA.data(), HL1, 8, xf_mul(xf_times100(xf_from(sv)), xf_from(r)), {0, 0}, 0, K);
    const double zd = sv * r;
    for (int l = 0; l <= 8; l++) {
      Q e = 0;
      double ed = 0;
      if (z < 16) {  // the reference's polynomial about the nearest table point
        const int i = (int)std::floor((double)(z * 100) + 0.5);
        const double *q = &t.besselH[((size_t)i * HL1 + l) * 6];
        const Q x = z - (Q)i / 100;
        for (int j = 5; j >= 0; j--) { e = e * x + q[j]; ed = std::fma(ed, zd - t.besselZ[i], q[j]); }
      } else {
        const Q a = (Q)0.5 / z;
        for (int j = l; j >= 0; j--) {
          e = e * (-a) + t.besselA[(size_t)l * AS + j];
          ed = std::fma(ed, -0.5 / zd, t.besselA[(size_t)l * AS + j]);
        }
        e *= a;
        ed *= 0.5 / zd;
      }
      wf[l] = std::fmax(wf[l], std::fabs((double)((K[l] - e) / e)));
      wx[l] = std::fmax(wx[l], std::fabs((double)((ed - e) / e)));
    }
  }
  double K0[16];
  fx_bessel_rows(t.besselX.data(), t.besselXA.data(), HL1, 8, {0, 0}, {0, 0}, 0, K0);
  for (int l = 1; l <= 8; l++) zero += K0[l];
  int worse = 0;
  for (int l = 0; l <= 8; l++) worse += wf[l] > wx[l];
  std::printf("%.3g %.3g %.3g %.3g %d %.3g %.3g %.3g %d %g %g\n", std::log2(we), std::log2(wd), std::log2(wr), wm, pack, wf[0],
              wf[2], wx[2], worse, K0[0], zero);
}
"""


def test_fixed_point_arithmetic(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(SRC)
    r = subprocess.run(["g++", "-O2", "-std=gnu++17", "-I", os.path.join(ROOT, "libecp_gb300", "csrc"), "-I",
                        os.path.join(ROOT, "include"), src, "-lquadmath", "-o", exe], capture_output=True, text=True)
    if r.returncode and "quadmath" in r.stderr:
        pytest.skip("no libquadmath on this machine")
    assert r.returncode == 0, r.stderr
    o = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    exp_bits, dbl_bits, rec_bits, mul_units, pack = float(o[0]), float(o[1]), float(o[2]), float(o[3]), int(o[4])
    assert exp_bits <= -58 and dbl_bits <= -52.95 and rec_bits <= -60
    assert mul_units <= 3 and pack == 0
    assert float(o[5]) <= 2 * 2.0 ** -53 and float(o[6]) <= float(o[7]) and int(o[8]) == 0, o
    assert float(o[9]) == 1.0 and float(o[10]) == 0.0
