"""The batched path's unit stages: a job cut into chunks by its scratch (here by
a request server's budget) gives bit for bit the values of one chunk, in every mode; primitive pairs of negative prefactor take the regrouped
small-grid kind and stay within the bar of the plain path; a contraction of 16
against 1 (parts and groups of one pair) and a single pair."""
import ctypes as ct

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


@pytest.mark.parametrize("mode_name", ["ECPGB_FP64", "ECPGB_FAST", "ECPGB_MIXED"])
@pytest.mark.parametrize("room", [0.95, 0.75])
def test_chunks_leave_results_unchanged(eg, mode_name, room):
    mode = getattr(eg, mode_name)
    s = W.batched_cluster(0, n_centres=4, n_basis_atoms=10)
    ref = eg.get_integrals_info(s, mode=mode)[1]
    with eg.Server(mode=mode, budget_bytes=8 << 30, slots=1) as sv:
        full = sv.wait(sv.submit(s))[2]["deviceBytes"]
    # the budget leaves part of the scratch the job would take
    with eg.Server(mode=mode, budget_bytes=int(full * room), slots=1) as sv:
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


def _noalloc(eg, s):
    L = eg.lib()
    L.ecpgb_getIntegrals_noalloc.argtypes = [ct.POINTER(eg.EcpgbSystem), ct.c_int, eg._D]
    I = np.zeros((s.dim, s.dim))
    assert L.ecpgb_getIntegrals_noalloc(ct.byref(eg.c_system(s)), s.dim, I.ctypes.data_as(eg._D)) in (0, 2)
    return I


PLAIN = {
    "example": lambda: W.example_like(0),
    "cluster": lambda: W.batched_cluster(3).subset(centres=[0, 3], basis_atoms=range(4)),
    "g_shells": lambda: W.mixed_batch(2, n_shells=8, n_centres=2),
    "L5_exponents_to_500": lambda: W.large_sweep(1, n_shells=10, n_centres=2),
    "on_the_centre": lambda: W.random_system(41, n_atoms=3, n_centres=3, lmax_basis=3, lmax_ecp=3),
    "reference_aborts": lambda: W.batched_cluster(0).subset(centres=[0], basis_atoms=[1, 6]),
    "never_converges": lambda: _with(W.random_system(26, n_atoms=2, n_centres=1, lmax_basis=1, lmax_ecp=2), tolerance=1e-300),
    "other_grid": lambda: _with(W.random_system(23, n_atoms=3, n_centres=2, lmax_basis=2, lmax_ecp=3, kmax=8),
                                largeGridOrder=8190, tolerance=1e-10, accuracy=1e-12),
}


def _with(s, **kw):
    s.nECP[::3] += 0.5
    for k, v in kw.items():
        setattr(s, k, v)
    return s


@pytest.mark.parametrize("name", list(PLAIN))
def test_plain_stages_equal_the_single_kernel_bit_for_bit(eg, name):
    """getIntegrals (the staged plain path) against the entry point that runs a
    unit per CTA with the reference's operations one by one."""
    s = PLAIN[name]()
    rc, I, _ = eg.get_integrals_info(s, mode=eg.ECPGB_FP64)
    assert np.array_equal(np.triu(I), np.triu(_noalloc(eg, s)))


@pytest.mark.parametrize("mode_name", ["ECPGB_FAST", "ECPGB_MIXED"])
@pytest.mark.parametrize("centres, atoms", [(1, 9), (1, 10), (1, 21), (2, 21)])
def test_job_sizes_on_both_sides_of_the_entry_rules(eg, mode_name, centres, atoms):
    """Primitive pairs: up to 9728 an entry is one pair, up to 58368 two warps
    take a large-grid entry; (1, 9) and (1, 10), (1, 21) and (2, 21) straddle the
    lines."""
    s = W.batched_cluster(5, n_centres=centres, n_basis_atoms=atoms)
    k = np.asarray(s.KBS, dtype=int)
    pairs = centres * (k.sum() ** 2 + (k ** 2).sum()) // 2
    assert (pairs <= 9728) == (atoms == 9) and (pairs <= 58368) == (centres == 1), pairs
    v0, o0, st0, _ = eg.raw_blocks(s, eg.ECPGB_FP64)
    v1, o1, st1, _ = eg.raw_blocks(s, getattr(eg, mode_name))
    assert np.array_equal(st0, st1) and np.array_equal(o0, o1)
    assert np.abs(v1 - v0).max() <= TOL_ABS


ODD = {
    "nan_coefficient": lambda s: s.dBS.__setitem__(0, np.nan),
    "infinite_ecp_coefficient": lambda s: s.dECP.__setitem__(1, np.inf),
    "growing_potential": lambda s: s.aECP.__setitem__(1, -0.01),
    "huge_coefficient": lambda s: s.dBS.__setitem__(0, 1e200),
    "high_power": lambda s: s.nECP.__setitem__(0, 24.0),
    "loose_accuracy": lambda s: setattr(s, "accuracy", 10.0),
}


@pytest.mark.parametrize("mode_name", ["ECPGB_FAST", "ECPGB_MIXED"])
@pytest.mark.parametrize("name", list(ODD))
def test_inputs_outside_the_integer_range_take_the_plain_stages(eg, mode_name, name):
    s = W.example_like(0)
    ODD[name](s)
    ref, got = eg.blocks(s, mode=eg.ECPGB_FP64), eg.blocks(s, mode=getattr(eg, mode_name))
    assert np.array_equal(ref[0], got[0]) and np.array_equal(ref[1], got[1], equal_nan=True)
    launches = []
    for mode in (eg.ECPGB_FP64, getattr(eg, mode_name)):
        job = eg.Job(s, mode=mode)
        launches.append(job.launches_per_run())
        job.close()
    assert launches[0] == launches[1]
