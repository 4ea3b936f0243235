"""The host tables with and without the batched path's fixed-point rows: an entry
point that runs the plain path only (ecpgb_getIntegrals_noalloc, libECP_init)
builds its tables on every call and leaves those rows out."""
import os
import subprocess

from tests.helpers import ROOT

SRC = r"""
#include "ecp_tables.cpp"
#include <cstdio>
using namespace ecpgb;
int main() {
  HostTables a, b, c;
  build_tables({5, 4, 1024, 1e-12, 1e-14, {}}, a);
  build_tables({5, 4, 1024, 1e-12, 1e-14, {}}, b, false);
  const bool left_out = b.besselX.empty() && b.besselXA.empty() && b.status == 0;
  const bool rest = a.besselH == b.besselH && a.besselA == b.besselA && a.besselT == b.besselT && a.shNorm == b.shNorm &&
                    a.omega == b.omega;
  bessel_fixed(b);
  std::printf("%d %d %d %d\n", left_out, rest, !a.besselX.empty(), a.besselX == b.besselX && a.besselXA == b.besselXA);
}
"""


def test_fixed_rows_are_built_apart(tmp_path):
    src, exe = str(tmp_path / "t.cpp"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["g++", "-O2", "-std=gnu++17", "-I", os.path.join(ROOT, "libecp_gb300", "csrc"), "-I",
                    os.path.join(ROOT, "include"), src, "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    assert out == ["1", "1", "1", "1"]
