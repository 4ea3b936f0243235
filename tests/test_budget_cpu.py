"""The request server's arithmetic on the host: what a job is said to hold within
a budget (ecpgb::job_device_bytes) never exceeds it while the scratch between the
unit stages can shrink, and a job is refused only where its other buffers alone
are above the budget."""
import ctypes as ct
import os
import subprocess

import pytest

from libecp_gb300 import workloads as W
from tests.helpers import ROOT

SRC = r"""
#include "ecp_host.h"
extern "C" int probe(const ecpgb_system *s, int mode, long long budget, long long *out) {
  ecpgb::Parsed P;
  if (ecpgb::parse_system(*s, P)) return -1;
  ecpgb::JobBytes need;
  size_t cap = 0;
  const bool ok = ecpgb::job_device_bytes(P, mode, (size_t)budget, &need, &cap);
  out[0] = (long long)need.total();
  out[1] = (long long)need.b[ecpgb::kJobBufs - 1];
  out[2] = (long long)cap;
  return ok;
}
"""


@pytest.fixture(scope="module")
def eg():
    import libecp_gb300
    libecp_gb300.lib()
    return libecp_gb300


@pytest.fixture(scope="module")
def probe(eg, tmp_path_factory):
    d = tmp_path_factory.mktemp("budget")
    src, so = str(d / "p.cpp"), str(d / "p.so")
    with open(src, "w") as f:
        f.write(SRC)
    lib = os.path.join(ROOT, "libecp_gb300")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(lib, "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include", src, "-L", lib, "-l:libecp_gb300.so",
                    "-Wl,-rpath," + lib, "-o", so], check=True)
    L = ct.CDLL(so)

    def run(s, mode, budget):
        out = (ct.c_longlong * 3)()
        cs = eg.c_system(s)
        rc = L.probe(ct.byref(cs), mode, ct.c_longlong(budget), out)
        assert rc >= 0
        return bool(rc), out[0], out[1], out[2]
    return run


SYSTEMS = {
    "example": lambda: W.example_like(0),
    "cluster": lambda: W.batched_cluster(0, n_centres=12, n_basis_atoms=10),
    "many_centres": lambda: W.batched_cluster(1, n_centres=60, n_basis_atoms=12, l_weights=(1.0,), kmax=1),
    "long_contractions": lambda: W.mixed_batch(2, n_shells=20, n_centres=3),
}


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("name", list(SYSTEMS))
def test_a_job_stays_within_its_budget(probe, name, mode):
    s = SYSTEMS[name]()
    ok, full, scratch, cap = probe(s, mode, 1 << 40)
    assert ok and scratch <= cap + 16
    other = full - scratch  # everything but the scratch
    for k in range(0, 20):
        budget = other + (full - other) * k // 19
        ok, need, scr, cap = probe(s, mode, budget)
        # within the budget, but where the scratch is at its smallest (one entry)
        assert ok and (need <= budget or scr > cap + 16), (k, need, budget, scr, cap)
    assert not probe(s, mode, other // 2)[0]
