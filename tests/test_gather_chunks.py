"""Node gathers of the scalar advection hand values from layer to layer inside a chunk: chunks of
one layer, with a remainder, and of the whole column, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kb,layers", [(4, 1), (4, 2), (4, 4), (8, 1), (8, 3), (8, 8), (11, 4)])
@pytest.mark.parametrize("mesh", ["channel", "coast"])
def test_chunks_of_layers(mesh, kb, layers):
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom
    from oracle.oracle import Oracle
    if mesh == "channel":
        case = cases.estuary_channel(nx=24, ny=6, kb=kb, lx=4800.0, ly=1200.0, IRAMP=10)
    else:
        case = cases.coastal_mesh(npts=600, kb=kb, lx=20000.0, ly=10000.0, seed=5, IRAMP=20)
    a, o = Fvcom(case), Oracle(case)
    a.set_tuning("col_layers", layers)
    a.run(4)
    o.run(4)
    for f in ("q2", "q2l", "t1", "s1", "km", "el", "u"):
        x, y = a.get(f), o.get(f)
        assert np.abs(x - y).max() <= 1e-10 * np.abs(y).max(), f
    a.close()
    o.close()
