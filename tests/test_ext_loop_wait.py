"""The resident external loop's grid barrier waits for a bounded number of polls.  Where a wait
runs out (here: none allowed) the kernel returns, the call reports FVG_ERR_TIMEOUT, every later
one does too, and setting the state and the clock again makes the model whole."""
import time

import numpy as np
import pytest

from tests import parity

pytestmark = pytest.mark.gpu
TIMEOUT = "status 5"
FIELDS = ("el", "ua", "va", "u", "t1", "s1", "q2", "km")


def _restore(src, dst):
    for n in parity.ALL + [b for pair in parity.MAPPED.values() for b in pair]:
        dst.set(n, src.get(n))
    dst.set_clock(*src.clock())


def _fails(call):
    from myfvcomcode_b200.engine import FvgError
    t = time.time()
    with pytest.raises(FvgError) as e:
        call()
    assert TIMEOUT in str(e.value) and "barrier" in str(e.value)
    assert time.time() - t < 5.0


def test_a_wait_that_runs_out_is_reported_until_the_state_is_set(small_channel):
    from myfvcomcode_b200.engine import Fvcom
    a, b = Fvcom(small_channel), Fvcom(small_channel)
    a.run(2)
    polls = a.get_tuning("ext_loop_polls")
    assert polls > 0
    a.set_tuning("ext_loop_polls", 0)
    _fails(lambda: a.run(3))
    a.set_tuning("ext_loop_polls", polls)
    clock = a.clock()
    _fails(lambda: a.run(1))
    _fails(a.internal_step)
    _fails(lambda: a.time_steps(1))
    assert a.clock() == clock  # a refused step is no step
    _restore(b, a)
    a.run(4)
    b.run(4)
    for f in FIELDS:
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()


def test_a_group_keeps_its_clocks_together(small_channel, small_coastal):
    from myfvcomcode_b200.engine import Fvcom, Group
    models = [Fvcom(c) for c in (small_coastal, small_channel, small_coastal)]
    fresh = [Fvcom(c) for c in (small_coastal, small_channel)]
    grp = Group(models)
    grp.run(1)
    polls = models[1].get_tuning("ext_loop_polls")
    models[1].set_tuning("ext_loop_polls", 0)
    _fails(lambda: grp.run(2))
    assert len({m.clock() for m in models}) == 1
    models[1].set_tuning("ext_loop_polls", polls)
    _fails(lambda: grp.run(1))
    assert len({m.clock() for m in models}) == 1
    # the models whose own waits did not run out stepped as ever
    fresh[0].run(3)
    for f in FIELDS:
        for m in (models[0], models[2]):
            assert np.array_equal(m.get(f), fresh[0].get(f)), f
    fresh[1].run(3)
    _restore(fresh[1], models[1])
    grp.run(2)
    for m in fresh:
        m.run(2)
    for m, ref in ((models[0], fresh[0]), (models[1], fresh[1]), (models[2], fresh[0])):
        for f in FIELDS:
            assert np.array_equal(m.get(f), ref.get(f)), f
    grp.close()
    for m in models + fresh:
        m.close()


def test_polls_are_checked(small_channel):
    from myfvcomcode_b200.engine import Fvcom, FvgError
    a = Fvcom(small_channel)
    with pytest.raises(FvgError):
        a.set_tuning("ext_loop_polls", -1)
    a.close()
