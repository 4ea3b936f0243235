"""Jobs on a GPU with little free memory: an allocation that fails (here by a
cudaMalloc that refuses sizes above a limit) costs chunks, not the call."""
import os
import subprocess
import sys

import pytest

from tests.helpers import ROOT

pytestmark = pytest.mark.gpu

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
static size_t limit(void) {
  const char *s = getenv("TEST_MALLOC_LIMIT");
  return s ? strtoull(s, 0, 10) : (size_t)-1;
}
int cudaMalloc(void **p, size_t n) {
  static int (*f)(void **, size_t);
  if (n > limit()) return 2; /* cudaErrorMemoryAllocation */
  if (!f) f = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMalloc");
  return f(p, n);
}
int cudaMallocAsync(void **p, size_t n, void *s) {
  static int (*f)(void **, size_t, void *);
  if (n > limit()) return 2;
  if (!f) f = (int (*)(void **, size_t, void *))dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMallocAsync");
  return f(p, n, s);
}
"""

SCRIPT = """
import os, sys
import numpy as np
import libecp_gb300 as eg
from libecp_gb300 import workloads as W
mode = getattr(eg, sys.argv[1])
s = W.batched_cluster(0, n_centres=8, n_basis_atoms=20)
# no buffer but the scratch is above the limit
os.environ["TEST_MALLOC_LIMIT"] = str(16 << 20)
I = eg.get_integrals_info(s, mode=mode)[1]
job = eg.Job(s, mode=mode)
job.run(2, flush_l2=False)
J = np.triu(job.matrix())
chunks = job.launches_per_run()
job.close()
with eg.Server(mode=mode, budget_bytes=8 << 30, slots=1) as sv:
    rc, K, _ = sv.wait(sv.submit(s))
del os.environ["TEST_MALLOC_LIMIT"]
job = eg.Job(s, mode=mode)
assert job.launches_per_run() < chunks, "the limit was not met"
job.close()
ref = eg.get_integrals_info(s, mode=mode)[1]
assert np.array_equal(I, ref) and np.array_equal(J, np.triu(ref)) and np.array_equal(K, np.triu(ref))
print("same")
"""


@pytest.mark.parametrize("mode", ["ECPGB_FP64", "ECPGB_FAST"])
def test_scratch_that_cannot_be_had(tmp_path, mode):
    src, so = str(tmp_path / "shim.c"), str(tmp_path / "shim.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", src, "-o", so, "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT, mode], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=ROOT, LD_PRELOAD=so))
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
