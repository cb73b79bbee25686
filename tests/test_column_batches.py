"""Column kernels that load a batch of layers (8, or 4 in VDIF_UV and BAROPG) before they work on
it: layer counts below, at and beside a batch, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb", [4, 5, 6, 9, 10, 17])
def test_layer_counts_beside_a_batch(kb):
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom
    from oracle.oracle import Oracle
    case = cases.coastal_mesh(npts=600, kb=kb, lx=20000.0, ly=10000.0, seed=5, IRAMP=20)
    a, o = Fvcom(case), Oracle(case)
    a.run(4)
    o.run(4)
    for f in ("el", "u", "v", "w", "wts", "ww", "rho1", "rho", "t1", "s1", "q2", "km"):
        x, y = a.get(f), o.get(f)
        assert np.abs(x - y).max() <= 1e-10 * np.abs(y).max(), f
    a.close()
    o.close()
