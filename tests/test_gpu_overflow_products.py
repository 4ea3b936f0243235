"""Small-grid points below the screen or outside the window, and primitive pairs of
prefactor 0, where a potential or a product is beyond FP64's range: infinity times 0 is
NaN, and the plain path's quadratures meet it as the single kernel's do."""
import ctypes as ct

import numpy as np
import pytest

from libecp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eg():
    import libecp_gb300
    libecp_gb300.lib()
    return libecp_gb300


# (ECP term, shells (l, primitives (coefficient, exponent)), their position).
# On a centre a pair of exponents 20 is below the screen from r = 0.92 on and in the
# window up to 1.27; r^100000 is infinite beyond 1.007.  At 30 the window of an
# exponent 20 is a few points, and 1e308 r^-2 infinite at the head's lower ones.
def _sp(prims):
    return [(l, prims) for l in range(2)]


CASES = {
    "screened_potential": ((1e5, 1.0, 1.0), _sp([(1.0, 20.0)]), 0.0),
    "infinite_potential": ((1e5, 1.0, 1.0), _sp([(1.0, 20.0)]), 0.1),
    "zero_coefficient": ((2.0, 1.7e308, 800.0), _sp([(1.0, 100.0), (0.0, 1e-3)]), 0.4),
    "outside_the_window": ((-2.0, 1e308, 0.0), [(0, [(1.0, 20.0)]), (2, [(1.0, 1.0), (1.0, 1e-3)])], 30.0),
    "infinite_prefactor": ((0.0, 1.0, 2.0), _sp([(1e160, 1.0)]), 0.7),
}


@pytest.mark.parametrize("name", CASES)
def test_products_beyond_range_equal_the_single_kernel(eg, name):
    term, shells, x = CASES[name]
    b = W._Builder()
    b.atom([0.0, 0.0, 0.0], ecp=[(l, [(0.0, 1.0, 1.0), term]) for l in range(2)])
    b.atom([x, 0.0, 0.0], shells=shells)
    s = b.build("overflowing_products")
    L = eg.lib()
    L.ecpgb_getIntegrals_noalloc.argtypes = [ct.POINTER(eg.EcpgbSystem), ct.c_int, eg._D]
    I = np.zeros((s.dim, s.dim))
    assert L.ecpgb_getIntegrals_noalloc(ct.byref(eg.c_system(s)), s.dim, I.ctypes.data_as(eg._D)) in (0, 2)
    for mode in (eg.ECPGB_FP64, eg.ECPGB_FAST):  # (such jobs run the plain stages)
        J = eg.get_integrals_info(s, mode=mode)[1]
        assert np.array_equal(np.triu(I), np.triu(J), equal_nan=True)
