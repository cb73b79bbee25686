"""A group's step is captured once; a change to one of its models after that (precision form,
tuning) takes effect in the group's next step as it does in the model's own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_group_follows_a_change_of_form(small_channel, small_coastal):
    from myfvcomcode_b200.engine import Fvcom, Group
    alone = [Fvcom(c) for c in (small_channel, small_coastal)]
    both = [Fvcom(c) for c in (small_channel, small_coastal)]
    grp = Group(both)
    grp.run(2)
    for m in alone:
        m.run(2)
    for m in (alone[1], both[1]):
        m.set_precision("fp32flux")
    grp.run(2)
    for m in alone:
        m.run(2)
    for a, b in zip(alone, both):
        for f in ("el", "ua", "u", "t1", "q2"):
            assert np.array_equal(a.get(f), b.get(f)), f
    for m in (alone[1], both[1]):
        m.set_precision("fp64")
        m.set_tuning("ext_loop", 0)
    grp.run(2)
    for m in alone:
        m.run(2)
    for a, b in zip(alone, both):
        for f in ("el", "ua", "u", "t1", "q2"):
            assert np.array_equal(a.get(f), b.get(f)), f
    grp.close()
    for m in alone + both:
        m.close()
