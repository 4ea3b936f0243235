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


@pytest.mark.parametrize("mode", [0, 1])
def test_the_smallest_scratch_is_one_unit(probe, mode):
    """40 centres on one shell pair of 16 x 16 primitives: a chunk may be a single
    unit of the 40."""
    b = W._Builder()
    shell = (4, [(0.1 + 0.05 * i, 0.05 * 1.7 ** i) for i in range(16)])
    for i in range(40):
        b.atom([0.5 * i, 0.1, 0.0], ecp=[(l, [(2.0, 1.0, 1.0)]) for l in range(4)], shells=[shell] if i == 0 else [])
    s = b.build("one_pair")
    ok, full, scratch, _ = probe(s, mode, 1 << 40)
    other = full - scratch
    one = -(-(scratch - 16) // 40)
    # the screening stage's and the plan's lists of 40 chunks take some more
    ok, need, scr, _ = probe(s, mode, other + one + 8192)
    assert ok and need <= other + one + 8192 and scr <= one + 4096
    ok, need, scr, _ = probe(s, mode, other)
    assert ok and scr <= one + 4096
