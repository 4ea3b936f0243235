"""Jobs of more units than a queue position holds are refused before any launch."""
import numpy as np
import pytest

from libecp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eg():
    import libecp_gb300
    libecp_gb300.lib()
    return libecp_gb300


def _s_shells(n_shells, n_centres):
    b = W._Builder()
    for i in range(n_centres):
        b.atom([0.1 * i, 0.0, 0.0], ecp=[(0, [(2.0, 1.0, 1.0)])],
               shells=[(0, [(1.0, 1.0)])] * (n_shells if i == 0 else 0))
    return b.build("many_units")


@pytest.mark.parametrize("mode_name", ["ECPGB_FP64", "ECPGB_FAST", "ECPGB_MIXED"])
def test_more_units_than_an_int_are_refused(eg, mode_name):
    s = _s_shells(2000, 1100)
    assert s.n_units > np.iinfo(np.int32).max
    with pytest.raises(RuntimeError, match="units"):
        eg.get_integrals_info(s, mode=getattr(eg, mode_name))
    with eg.Server(mode=getattr(eg, mode_name), budget_bytes=1 << 40, slots=1) as sv:
        with pytest.raises(RuntimeError, match="units"):
            sv.wait(sv.submit(s))
