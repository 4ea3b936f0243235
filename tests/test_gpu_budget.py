"""A request server whose budget holds each of two unlike jobs alone but not the
scratch of the first beside the buffers of the second: every request is answered,
with the values of the call made alone, and the slot stays within the budget."""
import os
import subprocess
import sys

import pytest

from tests.helpers import ROOT
from tests.test_budget_cpu import eg, probe  # noqa: F401 (fixtures)

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys
import numpy as np
import libecp_gb300 as eg
from libecp_gb300 import workloads as W
mode, slots = getattr(eg, sys.argv[1]), int(sys.argv[2])
scratchy = W.batched_cluster(0, n_centres=8, n_basis_atoms=20)
wide = W.batched_cluster(1, n_centres=36, n_basis_atoms=24, l_weights=(1.0,), kmax=1)
alone, held = [], []
for s in (scratchy, wide):
    alone.append(np.triu(eg.get_integrals_info(s, mode=mode)[1]))
    with eg.Server(mode=mode, budget_bytes=8 << 30, slots=1) as sv:
        held.append(sv.wait(sv.submit(s))[2]["deviceBytes"])
budget = max(held) + (1 << 16)
with eg.Server(mode=mode, budget_bytes=budget, slots=slots) as sv:
    for k in (0, 1, 0, 1, 1, 0):
        rc, I, info = sv.wait(sv.submit((scratchy, wide)[k]))
        assert rc in (0, 2) and np.array_equal(I, alone[k]), k
        assert info["deviceBytes"] <= budget and sv.stats()["deviceBytesHeld"] <= budget, (k, info, budget)
print("answered")
"""


@pytest.mark.parametrize("mode", ["ECPGB_FAST", "ECPGB_FP64"])
@pytest.mark.parametrize("slots", [1, 3])
def test_unlike_jobs_within_a_tight_budget(mode, slots):
    # in a process of its own: a server that stops answering ends with the timeout
    r = subprocess.run([sys.executable, "-c", SCRIPT, mode, str(slots)], cwd=ROOT, capture_output=True, text=True,
                       timeout=60, env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and "answered" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_chunks_that_begin_inside_a_pair_leave_results_unchanged(probe, mode):
    """25 centres on shells of up to 9 primitives: one pair's units take more than
    the smallest scratch (256 KiB or one unit), so chunks begin inside pairs; every
    value as in one chunk, within the budget where the scratch is above its
    smallest."""
    import numpy as np
    import libecp_gb300 as eg
    from libecp_gb300 import workloads as W
    rng = np.random.default_rng(3)
    b = W._Builder()
    for i in range(25):
        shells = [(l, W._shell(rng, l, k, 0.05, 20.0)[1]) for l, k in ((3, 9), (1, 4), (0, 1))] if i % 12 == 0 else []
        b.atom(rng.uniform(-4, 4, 3), ecp=W._ecp_channels(rng, 3, 3), shells=shells)
    s = b.build("inside_pairs")
    ref = np.triu(eg.get_integrals_info(s, mode=mode)[1])
    _, full, scratch, _ = probe(s, mode, 1 << 40)
    for part in (0.0, 0.01, 0.05, 0.2, 0.6):
        budget = full - scratch + int(part * scratch)
        with eg.Server(mode=mode, budget_bytes=budget, slots=1) as sv:
            rc, I, info = sv.wait(sv.submit(s))
        ok, need, scr, cap = probe(s, mode, budget)
        assert ok and info["deviceBytes"] == need and (need <= budget or scr > cap + 16), (part, info, need, budget)
        assert np.array_equal(I, ref), part
