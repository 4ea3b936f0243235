"""Magnitudes at the edges of what the batched path's integers take: at the largest
accepted coefficients the values are the plain path's to rounding, and where a product
of accepted inputs leaves FP64's range the plain stages decide (infinities and NaN
included), whichever mode was asked for."""
import numpy as np
import pytest

from libecp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eg():
    import libecp_gb300
    libecp_gb300.lib()
    return libecp_gb300


@pytest.mark.parametrize("mode_name", ["ECPGB_FAST"])  # (the mixed path's float pairs end at 1e38)
@pytest.mark.parametrize("basis, potential", [(1e60, 1e-10), (1e6, 1e100), (1e60, 1e-100)])
def test_largest_accepted_coefficients(eg, mode_name, basis, potential):
    s = W.example_like(0)
    s.dBS *= basis / np.abs(s.dBS).max()
    s.dECP *= potential / np.abs(s.dECP).max()
    # the convergence tests' tolerance follows the values, so both paths stop at the
    # same levels as with ordinary coefficients
    s.tolerance = min(1e100, 1e-12 * basis * basis * potential)  # (1e100: the largest accepted)
    v0, off, st0, _ = eg.raw_blocks(s, eg.ECPGB_FP64)
    v1, _, st1, _ = eg.raw_blocks(s, getattr(eg, mode_name))
    assert np.isfinite(v0).all() and np.array_equal(st0, st1)
    assert np.abs(v1 - v0).max() <= 1e-10 * np.abs(v0).max()


def _overflows(order=1024, n=16.0):
    """Diffuse s shells on a diffuse potential of a high power: each number is
    accepted, r^16 d c c is above 1e308.  (And r^-2 on a grid that has r = 0.)"""
    b = W._Builder()
    b.atom([0.0, 0.0, 0.0], ecp=[(l, [(n, d, 1e-12)]) for l, d in ((0, 1e100), (1, -1e100))])
    for i in range(2):
        b.atom([1.0 + i, 0.5, -0.3], shells=[(0, [(1e60, 1e-12 * (1 + i)), (3e59, 1e-11)])])
    return b.build("overflows", largeGridOrder=order)


@pytest.mark.parametrize("mode_name", ["ECPGB_FAST", "ECPGB_MIXED"])
@pytest.mark.parametrize("make", [_overflows, lambda: _overflows(8190, -2.0)])
def test_products_beyond_fp64_take_the_plain_stages(eg, mode_name, make):
    s = make()
    v0, _, st0, _ = eg.raw_blocks(s, eg.ECPGB_FP64)
    v1, _, st1, _ = eg.raw_blocks(s, getattr(eg, mode_name))
    assert np.array_equal(v0, v1, equal_nan=True) and np.array_equal(st0, st1)
