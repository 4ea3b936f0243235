"""The batched path's unit stages: a job cut into chunks by its scratch (here by
a request server's budget) gives bit for bit the values of one chunk, in both
batched modes; primitive pairs of negative prefactor take the regrouped
small-grid kind and stay within the bar of the plain path; a contraction of 16
against 1 (parts and groups of one pair) and a single pair."""
import numpy as np
import pytest

from libecp_gb300 import workloads as W
from oracle import oracle as O
from tests.helpers import TOL_ABS
from tests.test_gpu_parity import assert_blocks_match

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eg():
    import libecp_gb300
    libecp_gb300.lib()
    return libecp_gb300


@pytest.mark.parametrize("mode_name", ["ECPGB_FAST", "ECPGB_MIXED"])
@pytest.mark.parametrize("room", [0, 1 << 20])
def test_chunks_leave_results_unchanged(eg, mode_name, room):
    mode = getattr(eg, mode_name)
    s = W.batched_cluster(0, n_centres=4, n_basis_atoms=10)
    ref = eg.get_integrals_info(s, mode=mode)[1]
    with eg.Server(mode=mode, budget_bytes=8 << 30, slots=1) as sv:
        full = sv.wait(sv.submit(s))[2]["deviceBytes"]
    # the plain path's buffers are the batched path's but for the scratch
    with eg.Server(mode=eg.ECPGB_FP64, budget_bytes=8 << 30, slots=1) as sv:
        base = sv.wait(sv.submit(s))[2]["deviceBytes"]
    with eg.Server(mode=mode, budget_bytes=base + (1 << 20) + room, slots=1) as sv:
        rc, I, info = sv.wait(sv.submit(s))
    assert info["deviceBytes"] < full
    assert np.array_equal(I, np.triu(ref))


def test_negative_coefficients_and_contraction_edges(eg):
    rng = np.random.default_rng(8)
    b = W._Builder()
    b.atom([0.0, 0.0, 0.0], ecp=W._ecp_channels(rng, 3, 3))
    shells = []
    for l, k in ((0, 16), (1, 1), (2, 5), (3, 2)):
        _, prims = W._shell(rng, l, k, 0.05, 50.0)
        shells.append((l, [(d if i % 2 else -d, a) for i, (d, a) in enumerate(prims)]))
    b.atom([0.9, -0.4, 1.3], shells=shells[:2])
    b.atom([-1.1, 0.7, 0.2], shells=shells[2:])
    s = b.build("signs")
    rc, mo, do = O.oracle_blocks(s)
    meta, data = eg.blocks(s, mode=eg.ECPGB_FAST)
    assert_blocks_match(meta, data, mo, do)
    m0, d0 = eg.blocks(s)
    assert np.array_equal(m0, meta) and np.abs(d0 - data).max() <= TOL_ABS
