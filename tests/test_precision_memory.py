"""fvg_set_precision on a card without room for the FP32-flux form's scratch: the call fails,
the model stays in FP64 as it was, and a later call with room succeeds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_switch_without_room_leaves_the_model_whole():
    import torch
    from myfvcomcode_b200 import cases
    from myfvcomcode_b200.engine import Fvcom, FvgError
    case = cases.coastal_mesh(npts=20000, kb=21, lx=60000.0, ly=30000.0, seed=5, IRAMP=20)
    a, b = Fvcom(case), Fvcom(case)
    a.run(1)
    a.set_tuning("branches", 0)
    torch.cuda.synchronize()
    start = torch.cuda.mem_get_info()[0]
    b.set_precision("fp32flux")
    need = start - torch.cuda.mem_get_info()[0]
    for room in (need // 4, need // 2, need - (16 << 20)):
        fill = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        try:
            before = torch.cuda.mem_get_info()[0]
            with pytest.raises(FvgError):
                a.set_precision("fp32flux")
            assert a.get_precision() == "fp64"
            assert torch.cuda.mem_get_info()[0] == before
        finally:
            del fill
            torch.cuda.empty_cache()
    a.set_precision("fp32flux")
    a.set_precision("fp64")
    a.run(1)
    a.set_precision("fp32flux")
    a.run(2)
    b.set_precision("fp64")
    b.run(2)
    b.set_precision("fp32flux")
    b.run(2)
    for f in ("el", "u", "t1", "q2", "km"):
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()


def test_a_closure_without_room_leaves_the_model_whole():
    import os

    import torch
    from myfvcomcode_b200 import cases, closure
    from myfvcomcode_b200.engine import Fvcom, FvgError
    case = cases.coastal_mesh(npts=20000, kb=21, lx=60000.0, ly=30000.0, seed=5, IRAMP=20)
    net = closure.load(os.path.join(os.path.dirname(cases.__file__), "data", "closure_coastal50k_8seeds.npz"))
    a, b = Fvcom(case), Fvcom(case)
    a.set_tuning("branches", 0)
    torch.cuda.synchronize()
    start = torch.cuda.mem_get_info()[0]
    closure.attach(b, net)
    need = start - torch.cuda.mem_get_info()[0]
    for room in (need // 4, need - (2 << 20)):
        fill = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        try:
            before = torch.cuda.mem_get_info()[0]
            with pytest.raises(FvgError):
                closure.attach(a, net)
            assert torch.cuda.mem_get_info()[0] == before
        finally:
            del fill
            torch.cuda.empty_cache()
    closure.attach(a, net)
    a.run(3)
    b.run(3)
    for f in ("el", "u", "t1", "q2", "km"):
        assert np.array_equal(a.get(f), b.get(f)), f
    a.close()
    b.close()
