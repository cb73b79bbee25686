"""The scratch of a step's branches: one allocation for both precision forms, given back with
branches = 0, and left out where the card is short of memory instead of failing fvg_create."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def case():
    from myfvcomcode_b200 import cases
    return cases.coastal_mesh(npts=20000, kb=21, lx=60000.0, ly=30000.0, seed=5, IRAMP=20)


def _scratch_bytes(case):
    g = case["grid"]
    return 112 * (g["M"] + 1) * g["KB"]


SLACK = 6 << 20  # allocations come in pages of 2 MB


@pytest.mark.parametrize("precision", ["fp64", "fp32flux"])
def test_branches_off_gives_the_scratch_back(case, precision):
    from myfvcomcode_b200.engine import Fvcom
    a, b = Fvcom(case), Fvcom(case)
    for m in (a, b):
        m.set_precision(precision)
    a.run(2)
    assert a.get_tuning("branches") == 1
    before = _free()
    a.set_tuning("branches", 0)
    gain = _free() - before
    assert a.get_tuning("branches") == 0
    want = _scratch_bytes(case)
    assert want - SLACK <= gain <= 1.05 * want + SLACK, (gain, want)
    a.run(1)
    a.set_tuning("branches", 1)
    assert a.get_tuning("branches") == 1
    a.run(2)
    b.run(5)
    for f in ("el", "u", "t1", "q2", "km"):
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()


def test_group_survives_the_scratch_given_back(case, small_coastal):
    from myfvcomcode_b200.engine import Fvcom, Group
    a, b, other = Fvcom(case), Fvcom(case), Fvcom(small_coastal)
    grp = Group([a, other])
    grp.run(2)
    a.set_tuning("branches", 0)
    grp.run(2)
    b.run(4)
    for f in ("el", "u", "t1", "q2", "km"):
        assert np.array_equal(a.get(f), b.get(f)), f
    grp.close()
    for m in (a, b, other):
        m.close()


def test_a_card_short_of_memory_takes_no_branches(case):
    import torch
    from myfvcomcode_b200.engine import Fvcom
    ref = Fvcom(case)
    ref.run(2)
    start = _free()
    m = Fvcom(case)
    used = start - _free()
    m.close()
    # room for a model without the scratch, not for one with it
    room = used - _scratch_bytes(case) // 2
    fill = torch.empty(_free() - room, dtype=torch.uint8, device="cuda")
    try:
        m = Fvcom(case)
        assert m.get_tuning("branches") == 0
    finally:
        del fill
        torch.cuda.empty_cache()
    m.run(2)
    for f in ("el", "u", "t1", "q2", "km"):
        assert np.array_equal(m.get(f), ref.get(f)), f
    m.close()
    ref.close()
