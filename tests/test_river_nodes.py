"""Rivers that share a node (several at one node or cell, cells side by side): their temperature
and salinity are written in the order of the rivers, so the last one's stand, as in the oracle."""
import numpy as np
import pytest

from tests import parity
from tests.test_parity_gpu import routine_failures

pytestmark = pytest.mark.gpu


def _case(what):
    from myfvcomcode_b200 import cases, grid
    case = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10,
                                 river_location="node" if what == "node" else "edge")
    g, kbm1 = case["grid"], 5
    if what == "node":
        locs = [int(np.asarray(g["INODEQ"])[1])] * 5
    else:
        one = int(np.asarray(g["ICELLQ"])[1])
        # the head's cells, side by side, in an order that is not that of their nodes
        locs = [one] * 3 if what == "cell" else [one + 2, one - 2, one, one + 2]
    n = len(locs)
    grid._rivers(g, [dict(loc=q, dist=[1.0 / kbm1] * kbm1) for q in locs], g["RIVER_LOC"])
    case["forcing"] = dict(case["forcing"], qdis=np.linspace(10.0, 50.0, n), tdis=np.linspace(16.0, 12.0, n),
                           sdis=np.linspace(0.0, 3.0, n))
    return case


@pytest.mark.parametrize("what", ["node", "cell", "side_by_side"])
def test_the_last_river_of_a_node_stands(what):
    from myfvcomcode_b200.engine import Fvcom
    from oracle.oracle import Oracle
    case = _case(what)
    failures = routine_failures(case, 3)
    assert not failures, failures
    a, b = Fvcom(case), Oracle(case)
    a.run(6)
    b.run(6)
    bad = parity.compare(a, b, ["el", "ua", "va", "u", "v", "t1", "s1"], rtol=1e-9)
    assert not bad, bad
    a.close()
