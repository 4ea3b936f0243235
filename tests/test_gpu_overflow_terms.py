"""Potential terms whose D r^n is above FP64's range: the plain path leaves out terms
that cannot change the sum, and these are not among them (infinity times an
exponential that is 0 is NaN)."""
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


@pytest.mark.parametrize("n", [0.0, 1.0, 2.0])
def test_overflowing_terms_equal_the_single_kernel(eg, n):
    b = W._Builder()
    # r reaches 37: 5e305 r^2 is above 1.8e308 there, exp(-1369) is 0
    b.atom([0.0, 0.0, 0.0], ecp=[(l, [(0.0, 1.0, 1e-3), (n, 5e305, 1.0)]) for l in range(2)])
    b.atom([0.4, 0.1, -0.2], shells=[(l, [(1.0, 1e-3)]) for l in range(2)])
    s = b.build("overflowing_terms")
    L = eg.lib()
    L.ecpgb_getIntegrals_noalloc.argtypes = [ct.POINTER(eg.EcpgbSystem), ct.c_int, eg._D]
    I = np.zeros((s.dim, s.dim))
    assert L.ecpgb_getIntegrals_noalloc(ct.byref(eg.c_system(s)), s.dim, I.ctypes.data_as(eg._D)) in (0, 2)
    J = eg.get_integrals_info(s, mode=eg.ECPGB_FP64)[1]
    assert np.array_equal(np.triu(I), np.triu(J), equal_nan=True)
    assert n < 2.0 or np.isnan(I).any()  # the overflow was met
