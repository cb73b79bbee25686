"""fvg_kernels_per_step against the kernels that a profiler sees in replayed steps, over the
options that change a step's launches."""
import ctypes as C
import os

import pytest

pytestmark = pytest.mark.gpu

OPTIONS = {
    "plain": {},
    "fp32flux": dict(precision="fp32flux"),
    "launched_stages": dict(tuning=dict(ext_loop=0)),
    "general_stages": dict(tuning=dict(compact=0)),
    "one_order": dict(tuning=dict(branches=0)),
    "limited": dict(params=dict(LIMITER="LIMITED_1")),
    "limited_launched": dict(params=dict(LIMITER="LIMITED_1"), tuning=dict(ext_loop=0)),
    "limited_general": dict(params=dict(LIMITER="LIMITED_1"), tuning=dict(compact=0)),
    "limited_fp32flux": dict(params=dict(LIMITER="LIMITED_2"), precision="fp32flux"),
    "z_levels": dict(params=dict(BAROCLINIC_PRESSURE_GRADIENT="z coordinates")),
    "barotropic": dict(params=dict(BAROTROPIC=True)),
    "no_tracers": dict(params=dict(TEMPERATURE_ACTIVE=False, SALINITY_ACTIVE=False)),
    "staged": dict(tuning=dict(staged=2)),
    "closure": dict(closure=True),
    "final_split": dict(npts=20000, kb=14),
    "river": dict(channel=True),
}


def _kernels(model, steps):
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        model.run(steps)
        torch.cuda.synchronize()
    return sum(1 for e in prof.events() if "k_" in e.name)


@pytest.mark.parametrize("name", sorted(OPTIONS))
def test_kernels_per_step_is_what_a_step_launches(name):
    from myfvcomcode_b200 import cases, closure
    from myfvcomcode_b200.engine import Fvcom
    o = OPTIONS[name]
    if o.get("channel"):
        case = cases.estuary_channel(nx=24, ny=6, kb=6, lx=4800.0, ly=1200.0, IRAMP=10)
    else:
        npts = o.get("npts", 1500)
        lx = 20000.0 * (npts / 1500.0) ** 0.5
        case = cases.coastal_mesh(npts=npts, kb=o.get("kb", 7), lx=lx, ly=lx / 2, seed=7, IRAMP=20, **o.get("params", {}))
    m = Fvcom(case)
    m.set_precision(o.get("precision", "fp64"))
    for key, value in o.get("tuning", {}).items():
        m.set_tuning(key, value)
    if o.get("closure"):
        data = os.path.join(os.path.dirname(cases.__file__), "data", "closure_coastal50k_8seeds.npz")
        closure.attach(m, closure.load(data))
    m.run(1)
    m.lib.fvg_kernels_per_step.argtypes = [C.c_void_p]
    m.lib.fvg_kernels_per_step.restype = C.c_int32
    said = int(m.lib.fvg_kernels_per_step(m.h))
    assert _kernels(m, 3) == 3 * said
    m.close()
