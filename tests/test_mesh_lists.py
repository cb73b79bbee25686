"""Meshes whose edge and half-edge lists do not close around their cells -- an edge that lists
a node off its cells, two half-edges of a cell that part the same two nodes -- are stepped as
their lists say, as the oracle does it."""
import numpy as np
import pytest

from tests import parity
from tests.test_parity_gpu import routine_failures

pytestmark = pytest.mark.gpu


def _case(what, mesh="channel", **more):
    from myfvcomcode_b200 import cases
    if mesh == "coast":  # wetting and drying
        c = cases.coastal_mesh(npts=1500, kb=7, lx=20000.0, ly=10000.0, seed=7, IRAMP=20, **more)
    else:
        c = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10, **more)
    g = c["grid"]
    nv = np.asarray(g["NV"])
    if what in ("edge", "both"):
        # an interior edge whose first node is that of the cell beside the edge's first cell
        e = int(np.nonzero(np.asarray(g["ISBC"])[1:] == 0)[0][40]) + 1
        ia, ib = np.asarray(g["IEC"])[e]
        own = set(nv[ia]) | set(nv[ib])
        off = next(n for o in np.asarray(g["NBE"])[ia] if o > 0 and o != ib for n in nv[o] if n not in own)
        g["IENODE"][e, 0] = off
    if what in ("half_edge", "both"):
        ntrg, niec = np.asarray(g["NTRG"]), g["NIEC"]
        c0 = 77
        he = np.nonzero(ntrg == c0)[0]
        he = he[he > 0]
        niec[he[1]] = niec[he[0]]
    return c


@pytest.mark.parametrize("what", ["edge", "half_edge", "both"])
@pytest.mark.parametrize("mesh,ghost", [("channel", "GCN"), ("channel", "GCY1"), ("coast", "GCN")])
def test_routines_match_oracle(what, mesh, ghost):
    failures = routine_failures(_case(what, mesh, ghost_cells=ghost), 2)
    assert not failures, failures


@pytest.mark.parametrize("what", ["edge", "half_edge", "both"])
@pytest.mark.parametrize("mesh", ["channel", "coast"])
def test_steps_match_oracle(what, mesh):
    from myfvcomcode_b200.engine import Fvcom
    from oracle.oracle import Oracle
    case = _case(what, mesh)
    a, b = Fvcom(case), Oracle(case)
    assert a.get_tuning("ext_loop") == (1 if what == "half_edge" else 0)
    a.run(5)
    b.run(5)
    bad = parity.compare(a, b, ["el", "ua", "va", "u", "v", "t1", "s1", "q2"], rtol=1e-9)
    assert not bad, bad
    # the FP32-flux form takes the same lists
    c = Fvcom(case)
    c.set_precision("fp32flux")
    c.run(5)
    for f in ("el", "ua", "u"):
        x, y = c.get(f), a.get(f)
        assert np.abs(x - y).max() <= 1e-3 * np.abs(y).max(), f
    a.close()
    c.close()
