"""Sigma levels that differ from node to node (the library then reads the full arrays instead
of its table of levels) against the oracle, and the table against the full arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _vary(case):
    """Levels of a node spread by its own exponent; a cell's are the means of its nodes'."""
    g = case["grid"]
    M, KB = g["M"], g["KB"]
    s = (np.arange(KB) / (KB - 1))[None, :]
    e = 1.0 + 0.3 * np.sin(np.arange(M + 1))[:, None]
    z = -(s ** e)
    zz = np.zeros_like(z)
    zz[:, :-1] = 0.5 * (z[:, :-1] + z[:, 1:])
    zz[:, -1] = 2 * zz[:, -2] - zz[:, -3]
    dz, dzz = np.zeros_like(z), np.zeros_like(z)
    dz[:, :-1] = z[:, :-1] - z[:, 1:]
    dzz[:, :-1] = zz[:, :-1] - zz[:, 1:]
    for name, a in (("Z", z), ("ZZ", zz), ("DZ", dz), ("DZZ", dzz)):
        a[0] = 0.0
        g[name] = a
        c = np.zeros((g["N"] + 1, KB))
        nv = g["NV"]
        c[1:] = (a[nv[1:, 0]] + a[nv[1:, 1]] + a[nv[1:, 2]]) / 3.0
        g[name + "1"] = c
    return case


@pytest.mark.parametrize("mesh", ["channel", "coast"])
def test_levels_that_differ_per_node(mesh):
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom
    from oracle.oracle import Oracle
    if mesh == "channel":
        case = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10)
    else:
        case = cases.coastal_mesh(npts=1500, kb=7, lx=20000.0, ly=10000.0, seed=7, IRAMP=20)
    case = _vary(case)
    a, o = Fvcom(case), Oracle(case)
    a.run(5)
    o.run(5)
    for f in ("el", "u", "v", "w", "t1", "s1", "q2", "km"):
        x, y = a.get(f), o.get(f)
        assert np.abs(x - y).max() <= 1e-10 * np.abs(y).max(), f
    a.close()
    o.close()
