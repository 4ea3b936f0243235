"""Shells a little off an ECP centre: blocks that fall with powers of the distance
keep their relative precision in the batched and mixed paths.

Bar: both paths sum the same points of the same levels; a term differs by a few
units of 2^-53 (rows, exponentials, products: 2^-50 in all), and the potentials'
signs cancel at most two digits of a sum: 1e-13 of a block's largest value; 1e-12."""
import numpy as np
import pytest

from libecp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eg():
    import libecp_gb300
    libecp_gb300.lib()
    return libecp_gb300


def near_centre(delta):
    b = W._Builder()
    b.atom([0.0, 0.0, 0.0], ecp=[(l, [(2.0, c, a), (1.0, -0.6 * c, 2.3 * a)])
                                 for l, c, a in ((0, 3.0, 1.1), (1, -2.0, 0.7), (2, 1.5, 0.9), (3, 0.8, 0.6))])
    prims = [(0.7, 0.4), (0.5, 1.7), (0.3, 6.0)]
    b.atom([delta, -0.5 * delta, 0.25 * delta], shells=[(l, prims) for l in (0, 1, 2)])
    b.atom([1.1, -0.7, 0.9], shells=[(l, prims[:2]) for l in (0, 1, 2)])
    return b.build("near_centre")


@pytest.mark.parametrize("mode_name", ["ECPGB_FAST", "ECPGB_MIXED"])
@pytest.mark.parametrize("delta", [1e-9, 1e-7, 1e-6, 1e-5, 1e-4, 1e-3, 1e-2])
def test_small_blocks_keep_their_relative_precision(eg, mode_name, delta):
    s = near_centre(delta)
    v0, off, st0, _ = eg.raw_blocks(s, eg.ECPGB_FP64)
    v1, _, st1, _ = eg.raw_blocks(s, getattr(eg, mode_name))
    assert np.array_equal(st0, st1)
    l = np.asarray(s.lBS)
    # the units' order: atom pairs, then their shells (three each)
    pairs = [(3 * A + i, 3 * B + j) for A in range(2) for B in range(A, 2) for i in range(3) for j in range(3)
             if A < B or j >= i]
    small = 0
    for (i, j), o in zip(pairs, off):
        n = W.ncart(int(l[i])) * W.ncart(int(l[j]))
        for k in range(2):
            a, b = v0[o + k * n:o + (k + 1) * n], v1[o + k * n:o + (k + 1) * n]
            top = np.abs(a).max()
            small += 0 < top < 10 * delta
            assert np.abs(a - b).max() <= 1e-12 * top, (i, j, k, np.abs(a - b).max(), top)
    assert small or delta > 1e-3  # blocks that vanish with the distance are there
