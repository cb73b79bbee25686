"""The resident external loop against the launched stage kernels: the same FP64 results bit
for bit, on meshes around the loop's block sizes, with rivers, ghost cells, and dry cells
whose neighbours' flags it forms itself; in the FP32-flux form to FP32's rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("el", "elf", "elrk", "d", "dtfa", "egf", "el1", "elf1", "d1", "ua", "va", "uaf", "vaf", "uark", "uard",
          "vard", "advua", "pstx", "fluxobn", "uard_obcn", "iswetn", "iswetc", "iswetce", "u", "w", "t1", "q2")


def _case(name):
    from myfvcomcode_b200 import cases
    if name == "channel_node_river":
        return cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10)
    if name == "channel_edge_river":
        return cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10, river_location="edge")
    if name == "channel_wide":  # 148 blocks of 128 threads are not enough: the next block size
        return cases.estuary_channel(nx=170, ny=60, kb=4, lx=34000.0, ly=12000.0, IRAMP=10)
    ghost = name == "coast_ghost"
    npts = {"coast_large": 25000}.get(name, 1500)
    more = {"coast_limited_1": dict(LIMITER="LIMITED_1"), "coast_limited_2": dict(LIMITER="LIMITED_2")}.get(name, {})
    return cases.coastal_mesh(npts=npts, kb=5, lx=20000.0, ly=10000.0, seed=7, IRAMP=2, dte=0.5 if npts > 2000 else 2.0,
                              ghost_cells="GCY1" if ghost else "GCN", **more)


@pytest.mark.parametrize("name", ["channel_node_river", "channel_edge_river", "channel_wide", "coast", "coast_ghost",
                                  "coast_large", "coast_limited_1", "coast_limited_2"])
def test_resident_loop_equals_launched_loop(name):
    from myfvcomcode_b200.engine import Fvcom
    case = _case(name)
    a, b = Fvcom(case), Fvcom(case)
    b.set_tuning("ext_loop", 0)
    assert a.get_tuning("ext_loop") == 1 and b.get_tuning("ext_loop") == 0
    a.run(8)
    b.run(8)
    for f in FIELDS:
        assert np.array_equal(a.get(f), b.get(f)), f
    # the packed stages against the general stage kernels
    c = Fvcom(case)
    c.set_tuning("compact", 0)
    c.run(8)
    for f in FIELDS:
        assert np.array_equal(b.get(f), c.get(f)), f
    c.close()
    # one step without the graph
    a.use_graph(False)
    a.run(1)
    b.run(1)
    assert np.array_equal(a.get("ua"), b.get("ua"))
    a.close()
    b.close()


@pytest.mark.parametrize("name", ["channel_node_river", "coast"])
def test_resident_loop_fp32_flux(name):
    # 40 stages of FP32 fluxes whose viscosity products are rounded once more: a few 1e-7
    # of a flux, which is a small part of a stage's change
    from myfvcomcode_b200.engine import Fvcom
    case = _case(name)
    a, b = Fvcom(case), Fvcom(case)
    for m in (a, b):
        m.set_precision("fp32flux")
    b.set_tuning("ext_loop", 0)
    assert a.get_tuning("ext_loop") == 1
    a.run(4)
    b.run(4)
    for f in ("el", "ua", "va", "u", "t1"):
        x, y = a.get(f), b.get(f)
        assert np.abs(x - y).max() <= 1e-5 * np.abs(y).max(), f
    a.close()
    b.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32flux"])
def test_branches_equal_one_order(precision):
    from myfvcomcode_b200.engine import Fvcom, Group
    models = [Fvcom(_case("coast")) for _ in range(3)]
    for m in models:
        m.set_precision(precision)
    models[1].set_tuning("branches", 0)
    assert [m.get_tuning("branches") for m in models] == [1, 0, 1]
    models[0].run(6)
    models[1].run(6)
    grp = Group([models[2]])
    grp.run(6)
    for f in FIELDS + ("v", "s1", "km", "kh", "uf", "rho", "wubot", "tps"):
        for m in (models[0], models[2]):
            assert np.array_equal(m.get(f), models[1].get(f)), f
    # plain launches on the same streams
    models[0].use_graph(False)
    models[0].run(2)
    models[1].run(2)
    assert np.array_equal(models[0].get("t1"), models[1].get("t1"))
    grp.close()
    for m in models:
        m.close()
