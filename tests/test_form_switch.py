"""What a step in the FP32-flux form leaves in the handle's scratch does not reach a later step
in FP64, whatever the values were: a run that went wrong, its state set again and the form
changed back, continues as a model that never left FP64."""
import numpy as np
import pytest

from tests import parity

pytestmark = pytest.mark.gpu


def _restore(src, dst):
    names = [n for n in parity.ALL] + [b for pair in parity.MAPPED.values() for b in pair]
    for n in names:
        dst.set(n, src.get(n))
    dst.set_clock(*src.clock())


@pytest.mark.parametrize("ghost", ["GCN", "GCY1"])
def test_fp64_after_a_broken_fp32_run(ghost):
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom
    case = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10, ghost_cells=ghost)
    a, b = Fvcom(case), Fvcom(case)
    b.set_precision("fp32flux")
    ua = b.get("ua")
    ua[1] = np.nan
    b.set("ua", ua)
    b.run(1)
    assert np.isnan(b.get("ua")[1])
    b.set_precision("fp64")
    _restore(a, b)
    a.run(3)
    b.run(3)
    for f in ("el", "ua", "va", "u", "v", "w", "t1", "s1", "q2", "km", "viscofm"):
        assert np.isfinite(a.get(f)).all(), f
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()
