"""The end of the internal step as one kernel and, from half a million cells x levels on, as a
node kernel and a cell kernel: both sides of that size against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,kb", [(9000, 23), (13000, 23)])
def test_end_of_step(npts, kb):
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom
    from oracle.oracle import Oracle
    case = cases.coastal_mesh(npts=npts, kb=kb, lx=60000.0, ly=30000.0, seed=5, IRAMP=20)
    assert (case["grid"]["N"] * kb >= 500000) == (npts == 13000)
    a, o = Fvcom(case), Oracle(case)
    a.run(2)
    o.run(2)
    for f in ("t", "s", "rho", "rho1", "km1", "u", "v", "t1", "s1", "et1", "dt1"):
        x, y = a.get(f)[1:], o.get(f)[1:]  # entity 0 is no cell or node
        assert np.abs(x - y).max() <= 1e-10 * np.abs(y).max(), f
    a.close()
    o.close()
