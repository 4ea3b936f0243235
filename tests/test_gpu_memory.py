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


SHARED = """
import ctypes as ct, sys
import numpy as np
import libecp_gb300 as eg
from libecp_gb300 import workloads as W
rt = ct.CDLL("libcudart.so.13")
def free_bytes():
    f, t = ct.c_size_t(0), ct.c_size_t(0)
    assert rt.cudaMemGetInfo(ct.byref(f), ct.byref(t)) == 0
    return f.value
mode = getattr(eg, sys.argv[1])
small, large = (W.batched_cluster(0, n_centres=8, n_basis_atoms=n) for n in (12, 20))
eg.get_integrals_info(W.batched_cluster(0, n_centres=1, n_basis_atoms=3), mode=mode)
jobs = [eg.Job(small, mode=mode)]
def run(job):
    job.run(1, flush_l2=False)
    return job.matrix()
first = run(jobs[0])
f0 = free_bytes()
job = eg.Job(large, mode=mode)
run(job)
assert free_bytes() < f0 - (50 << 20)  # grown by 62 MB (batched) or more
job.close()
jobs[0].close()  # the last one gives the scratch back
assert free_bytes() > f0 - (8 << 20)
jobs[0] = eg.Job(small, mode=mode)
assert np.array_equal(run(jobs[0]), first)
jobs.append(eg.Job(large, mode=mode))  # the scratch grows under the first job's captured graph
second = run(jobs[1])
assert np.array_equal(run(jobs[0]), first)
f0 = free_bytes()
for _ in range(4):
    jobs.append(eg.Job(large, mode=mode))
per_job = (f0 - free_bytes()) / 4
assert all(np.array_equal(run(j), second) for j in jobs[2:])
assert np.array_equal(eg.get_integrals_info(large, mode=mode)[1], second)
assert np.array_equal(run(jobs[0]), first) and np.array_equal(run(jobs[1]), second)
for j in jobs:
    j.close()
# inputs and work arrays are 18 MB, the scratch 99 (batched) or 174 MB (plain)
assert per_job <= 40 << 20, per_job
print("shared")
"""


@pytest.mark.parametrize("mode", ["ECPGB_FP64", "ECPGB_FAST"])
def test_resident_jobs_share_the_scratch(mode):
    r = subprocess.run([sys.executable, "-c", SHARED, mode], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and "shared" in r.stdout, r.stderr[-2000:]
