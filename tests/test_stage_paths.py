"""Paths of the external loop that its other tests do not take: the launched stage kernels with
and without evict-first loads and walking threads, the FP32-flux form in each block shape of the
resident loop and with ghost cells, and lists longer than a thread of the loop keeps (four
rivers at a node or a cell, three open-boundary entries of a cell), and meshes that the packed
records do not fit."""
import numpy as np
import pytest

from tests import parity

pytestmark = pytest.mark.gpu

STATE = ("el", "elf", "d", "egf", "el1", "d1", "ua", "va", "uark", "uard", "vard", "advua", "pstx", "fluxobn", "uard_obcn",
         "iswetn", "iswetc", "iswetce", "u", "w", "t1", "s1", "q2")


@pytest.fixture(scope="module")
def large():
    from myfvcomcode_b200 import cases
    return cases.coastal_mesh(npts=20000, kb=7, lx=60000.0, ly=30000.0, seed=5, IRAMP=20)


@pytest.mark.parametrize("precision,limiter", [("fp64", "LIMITED_NO"), ("fp64", "LIMITED_1"), ("fp32flux", "LIMITED_NO")])
def test_launched_stages_walk_and_hint_bitwise(large, precision, limiter):
    from myfvcomcode_b200.engine import Fvcom
    case = dict(large, params=dict(large["params"], LIMITER=limiter))
    assert case["grid"]["N"] > 2 * 128 * 148
    a, b = Fvcom(case), Fvcom(case)
    for m in (a, b):
        m.set_precision(precision)
        m.set_tuning("ext_loop", 0)
    a.set_tuning("ext_grid", 1)  # each thread walks two to three cells
    b.set_tuning("ext_grid", 0)
    b.set_tuning("stream_hints", 0)
    a.run(3)
    b.run(3)
    for f in STATE:
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()


@pytest.mark.parametrize("cells_per_sm", ["half_block", "block", "large_block"])
def test_fp32_resident_loop_in_each_shape(cells_per_sm, large):
    # The two loops differ in the rounding of FP32 fluxes (a few 2^-24 of a flux, which is a small
    # part of a stage's change), over the forty stages of one step.
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom
    case = {"half_block": lambda: cases.estuary_channel(nx=90, ny=60, kb=4, lx=18000.0, ly=12000.0, IRAMP=10),
            "block": lambda: cases.estuary_channel(nx=170, ny=60, kb=4, lx=34000.0, ly=12000.0, IRAMP=10),
            "large_block": lambda: large}[cells_per_sm]()
    n = -(-case["grid"]["N"] // 148)
    assert {"half_block": 0, "block": 128, "large_block": 256}[cells_per_sm] < n <= {"half_block": 128, "block": 256,
                                                                                    "large_block": 384}[cells_per_sm]
    a, b = Fvcom(case), Fvcom(case)
    for m in (a, b):
        m.run(4)
        m.set_precision("fp32flux")
    b.set_tuning("ext_loop", 0)
    assert a.get_tuning("ext_loop") == 1 and a.get_tuning("compact") == 1
    a.run(1)
    b.run(1)
    for f in ("el", "ua", "va", "advua", "pstx", "d1"):
        x, y = a.get(f), b.get(f)
        assert np.abs(x - y).max() <= 1e-5 * np.abs(y).max(), f
    a.close()
    b.close()


@pytest.mark.parametrize("ghost", ["GCY1", "GCY2"])
@pytest.mark.parametrize("mesh", ["channel", "coast"])
def test_fp32_with_ghost_cells(mesh, ghost):
    # One step from a state that FP64 reached: the general, the packed and the resident stages
    # differ by the rounding of FP32 fluxes, some 1e-6 of what the step changes; a ghost
    # velocity taken wrongly changes a boundary cell's advection as a whole.
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom
    if mesh == "channel":
        case = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10, ghost_cells=ghost)
    else:
        case = cases.coastal_mesh(npts=1500, kb=5, lx=20000.0, ly=10000.0, seed=7, IRAMP=2, ghost_cells=ghost)
    models = [Fvcom(case) for _ in range(3)]
    for m in models:
        m.run(12)
        m.set_precision("fp32flux")
    models[1].set_tuning("ext_loop", 0)
    models[2].set_tuning("compact", 0)
    assert [m.get_tuning("ext_loop") for m in models] == [1, 0, 0]
    assert [m.get_tuning("compact") for m in models] == [1, 1, 0]
    before = {f: models[0].get(f) for f in ("el", "ua", "va")}
    for m in models:
        m.run(1)
    for f in ("el", "ua", "va"):
        ref = models[2].get(f)
        change = np.abs(ref - before[f]).max()
        for m in models[:2]:
            assert np.abs(m.get(f) - ref).max() <= 1e-3 * change, f
    for m in models:
        m.close()


def _rivers(location, n):
    from myfvcomcode_b200 import cases, grid
    case = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10, river_location=location)
    g, kbm1 = case["grid"], 5
    loc = int(np.asarray(g["INODEQ" if location == "node" else "ICELLQ"])[1])
    grid._rivers(g, [dict(loc=loc, dist=[1.0 / kbm1] * kbm1)] * n, location)
    case["forcing"] = dict(case["forcing"], qdis=np.linspace(10.0, 50.0, n), tdis=np.linspace(12.0, 16.0, n),
                           sdis=np.linspace(3.0, 0.0, n))
    return case


def _three_obc_entries():
    from myfvcomcode_b200 import cases
    case = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10)
    g = case["grid"]
    g["ADJC_OBC"][2:5, 0] = g["ADJC_OBC"][3, 0]
    assert (np.asarray(g["NADJC_OBC"])[2:5] >= 1).all()
    return case


@pytest.mark.parametrize("what", ["rivers_at_a_node", "rivers_at_a_cell", "open_boundary"])
def test_long_lists(what):
    from myfvcomcode_b200.engine import Fvcom
    from oracle.oracle import Oracle
    case = {"rivers_at_a_node": lambda: _rivers("node", 4), "rivers_at_a_cell": lambda: _rivers("edge", 4),
            "open_boundary": _three_obc_entries}[what]()
    models = [Fvcom(case) for _ in range(3)]
    models[1].set_tuning("ext_loop", 0)
    models[2].set_tuning("compact", 0)
    assert [m.get_tuning("ext_loop") for m in models] == [1, 0, 0]
    ora = Oracle(case)
    for m in models + [ora]:
        m.run(6)
    for f in STATE:
        for m in models[:2]:
            assert np.array_equal(m.get(f), models[2].get(f)), f
    assert np.isfinite(ora.get("ua")).all() and np.abs(ora.get("ua")).max() > 0
    bad = parity.compare(models[0], ora, ["el", "ua", "va", "u", "v", "t1", "s1"], rtol=1e-9)
    assert not bad, bad
    for m in models:
        m.close()


@pytest.mark.parametrize("metric", ["DLTXC", "XIJC", "DLTYE", "EPOR"])
def test_metrics_of_their_own_take_the_general_stages(metric):
    # a mesh whose edge metrics are not those of its coordinates, or whose masks are not 0 or 1
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom
    from tests.test_parity_gpu import routine_failures
    case = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10)
    a = case["grid"][metric]
    a[50] = 0.5 if metric == "EPOR" else a[50] + 1e-3
    m = Fvcom(case)
    assert m.get_tuning("ext_loop") == 0
    m.set_precision("fp32flux")
    assert m.get_tuning("compact") == 0
    m.close()
    failures = routine_failures(case, 2)
    assert not failures, failures
    from oracle.oracle import Oracle
    x, y = Fvcom(case), Oracle(case)
    x.run(5)
    y.run(5)
    bad = parity.compare(x, y, ["el", "ua", "va", "u", "v", "t1", "s1"], rtol=1e-9)
    assert not bad, bad
    x.close()
