"""The work that a user of this framework has it do, as timed cases.

A model run is a loop of internal steps (``Fvcom.run`` / ``Fvcom.internal_step``) between
output times, at which the history fields come back to host memory; a coupled program
sets the wind and reads the surface back every step; an ensemble steps several models as
one union model or one group; the learned closure is trained and evaluated on the device.
Each case makes its mesh once (it does not depend on the seed), a mid-run state from the
seed -- tide, wind, waves on the surface, currents, stratification with anomalies,
turbulence above its floor -- and the model that holds it.

``draw`` gives further cases of the same ranges: estuary channels from a few hundred
nodes, coastal meshes and unions of members up to 200,000 nodes and 40 layers, both
precisions, the optional schemes, and network sizes.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

from myfvcomcode_b200 import cases as fvcases
from myfvcomcode_b200 import closure, ensemble
from myfvcomcode_b200.abi import wind_stress
from myfvcomcode_b200.engine import Fvcom, Group, Mlp
from myfvcomcode_b200.startup import dens2

# History fields that come back at an output time.  The plain form returns them as the
# FP64 state holds them; the FP32-flux form as history files store them (single precision).
FIELDS = ("el", "ua", "va", "u", "v", "t1", "s1", "q2", "km")
CLOSURE = os.path.join(os.path.dirname(os.path.abspath(fvcases.__file__)), "data", "closure_coastal50k_8seeds.npz")


def listed():
    return [
        # the smallest call: a regression-sized channel driven step by step by a coupled host
        # program that reads the surface back each time
        dict(name="channel_coupled", kind="channel", nx=24, ny=6, kb=6, river="edge", precision="fp64",
             option="plain", call="coupled", steps=1),
        # the idealised estuary channel as specified (2,121 nodes, 10 layers), the everyday
        # plain run between outputs
        dict(name="channel_run", kind="channel", nx=100, ny=20, kb=11, river="node", precision="fp64",
             option="plain", call="run", steps=10),
        # a small wet/dry coast with the momentum limiter and surface heating switched on
        dict(name="coast_limited_heated", kind="coast", npts=1500, kb=7, members=1, precision="fp64",
             option="limited_heating", call="run", steps=10),
        # a regional mesh with ghost cells and an odd layer count, plain FP64
        dict(name="coast_ghost", kind="coast", npts=6000, kb=24, members=1, precision="fp64", option="ghost",
             call="run", steps=10),
        # a regional mesh in the FP32-flux form
        dict(name="coast_f32", kind="coast", npts=20000, kb=21, members=1, precision="fp32flux", option="plain",
             call="run", steps=10),
        # the 50k-node, 30-layer coastal mesh, plain FP64: production-sized runs
        dict(name="coast50k_fp64", kind="coast", npts=50000, kb=31, members=1, precision="fp64", option="plain",
             call="run", steps=6),
        # the same mesh in the FP32-flux form
        dict(name="coast50k_f32", kind="coast", npts=50000, kb=31, members=1, precision="fp32flux",
             option="plain", call="run", steps=10),
        # the same mesh coupled: new wind in and the surface out every step
        dict(name="coast50k_coupled", kind="coast", npts=50000, kb=31, members=1, precision="fp32flux",
             option="plain", call="coupled", steps=3),
        # four perturbed members as one union model, 200,000 nodes: the largest plain run
        dict(name="union200k_fp64", kind="coast", npts=50000, kb=31, members=4, precision="fp64",
             option="plain", call="run", steps=5),
        # a group in one graph: members of the coastal mesh with FP32 fluxes and the learned
        # closure beside members of the estuary channel (meshes of uneven size)
        dict(name="group_closure", kind="group", npts=50000, kb=31, members=2, channels=16, call="group", steps=5),
        # training the closure's network for an epoch
        dict(name="mlp_train", kind="train", n=262144, batch=4096, epochs=1),
        # evaluating it on a large set of samples
        dict(name="mlp_forward", kind="forward", n=1000003),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("channel", "coast", "train", "forward"), (4, 9, 1, 1))[0]
    if kind == "train":
        return dict(kind="train", n=_log_uniform(rng, 20000, 262144), batch=rng.choice((512, 1000, 4096)), epochs=1)
    if kind == "forward":
        return dict(kind="forward", n=_log_uniform(rng, 1000, 1000003))
    precision = rng.choice(("fp64", "fp32flux"))
    call, steps = rng.choice((("run", 5), ("run", 10), ("coupled", 3)))
    if kind == "channel":
        return dict(kind="channel", nx=_log_uniform(rng, 16, 200), ny=_log_uniform(rng, 5, 40), kb=rng.randint(5, 21),
                    river=rng.choice(("node", "edge")), precision=precision, option="plain", call=call, steps=steps)
    # single meshes up to 24,000 nodes, and unions of members of such a mesh above
    nodes = _log_uniform(rng, 800, 200000)
    members = -(-nodes // 24000)
    option = rng.choices(("plain", "limited_heating", "ghost", "zlevel"), (7, 1, 1, 1))[0] if members == 1 else "plain"
    return dict(kind="coast", npts=nodes // members, kb=rng.randint(7, 31 if members > 1 else 41), members=members,
                precision=precision, option=option, call=call, steps=steps)


# --------------------------------------------------------------------------------------
# meshes and states
# --------------------------------------------------------------------------------------
_MESH = {}


def _mesh(case):
    """The case dictionary of a mesh and its options, made once in a process."""
    keys = ("kind", "nx", "ny", "river") if case["kind"] == "channel" else ("kind", "npts", "members", "option")
    key = tuple(case.get(k) for k in keys) + (case["kb"],)
    if key in _MESH:
        return _MESH[key]
    if case["kind"] == "channel":
        made = fvcases.estuary_channel(nx=case["nx"], ny=case["ny"], kb=case["kb"], lx=200.0 * case["nx"],
                                       ly=200.0 * case["ny"], river_location=case["river"])
    elif case["members"] > 1:
        base = _mesh(dict(case, members=1))
        made = ensemble.union_case(base, ensemble.perturbed_members(base, case["members"], seed=5))
    else:
        npts, option = case["npts"], case["option"]
        # about 320 m between nodes below 50,000 nodes, the default box above
        lx = 200000.0 if npts >= 50000 else max(20000.0, 200000.0 * math.sqrt(npts / 200000.0))
        more = {}
        if option == "limited_heating":
            more = dict(LIMITER="LIMITED_1", HEATING_ON=True)
        elif option == "zlevel":
            more = dict(BAROCLINIC_PRESSURE_GRADIENT="z coordinates")
        made = fvcases.coastal_mesh(npts=npts, kb=case["kb"], lx=lx, ly=lx / 2, seed=1234,
                                    ghost_cells="GCY1" if option == "ghost" else "GCN", **more)
        if option == "limited_heating":
            made["forcing"]["heat"] = {"swrad": 400.0, "wtsurf": 250.0}
    _MESH[key] = made
    return made


def _waves(r, x, y, n=4):
    """A smooth field of order one over the mesh: a few long waves."""
    lx, ly = float(x.max() - x.min()) + 1.0, float(y.max() - y.min()) + 1.0
    f = np.zeros_like(x)
    for _ in range(n):
        kx, ky = r.uniform(-2.0, 2.0, 2)
        f += np.cos(2 * np.pi * (kx * x / lx + ky * y / ly) + r.uniform(0.0, 2 * np.pi)) / n
    return f


def _n2e(g, a):
    nv = g["NV"]
    out = np.zeros((g["N"] + 1,) + a.shape[1:])
    out[1:] = (1.0 / 3.0) * (a[nv[1:, 0]] + a[nv[1:, 1]] + a[nv[1:, 2]])
    return out


def _forced(base, r):
    """``base`` with the seed's wind and tidal phase, and the start of the run's clock."""
    c = dict(base, forcing=dict(base["forcing"]))
    f = c["forcing"]
    N = c["grid"]["N"]
    speed, head = r.uniform(7.0, 8.5), r.uniform(0.0, 2 * np.pi)
    sx, sy = fvcases.simple_drag(np.full(N + 1, speed * np.cos(head)), np.full(N + 1, speed * np.sin(head)))
    f["wind"] = {"kind": "field", "sx": sx, "sy": sy}
    phase = r.uniform(0.0, 360.0)
    f["tide"] = dict(f["tide"], phai=np.asarray(f["tide"]["phai"]) + phase)
    return c, 720, float(20.0 * r.integers(720, 4000))


def _state(c, r, iint, t0):
    """A mid-run state: FVCOM's arrays by name, consistent with one another."""
    g, p = c["grid"], c["params"]
    M, N, KB = g["M"], g["N"], g["KB"]
    h, md, tide = g["H"], p["MIN_DEPTH"], c["forcing"]["tide"]
    ramp = math.tanh(iint / p["IRAMP"])
    level = sum(float(np.mean(tide["apt"][:, j])) * math.cos(2 * math.pi * t0 / float(tide["period"][j]) -
                                                             math.radians(float(np.mean(tide["phai"][:, j]))))
                for j in range(len(tide["period"]))) * ramp
    x, y, xc, yc = g["VX"], g["VY"], g["XC"], g["YC"]
    el = level + 0.05 * _waves(r, x, y)
    iswetn, iswetc = np.ones(M + 1, np.int32), np.ones(N + 1, np.int32)
    if p["WETTING_DRYING_ON"]:
        nv, ntve, nbve = g["NV"], g["NTVE"], g["NBVE"]
        iswetn[1:][(h[1:] + el[1:] - md) < 1.0e-5] = 0
        e3, h3 = el[nv[1:]], h[nv[1:]]
        iswetc[1:][(e3.max(axis=1) + h3.min(axis=1) - md) < 1.0e-5] = 0
        ring = np.arange(nbve.shape[1])[None, :] < ntve[:, None]
        iswetn[1:][((iswetc[nbve] * ring).sum(axis=1) == 0)[1:]] = 0
        el = np.maximum(el, -h + md)
    el1 = _n2e(g, el)
    d, d1 = h + el, g["H1"] + el1
    st = dict(el=el, elf=el, et=el, el1=el1, elf1=el1, et1=el1, d=d, dt=d, dtfa=d, d1=d1, dt1=d1,
              iswetn=iswetn, iswetnt=iswetn, iswetc=iswetc, iswetct=iswetc, iswetce=iswetc)
    wetc = iswetc.astype(np.float64)
    ua, va = 0.1 * _waves(r, xc, yc) * wetc, 0.1 * _waves(r, xc, yc) * wetc
    zz, zz1, z = g["ZZ"][:, :KB], g["ZZ1"], g["Z"]
    shear = np.zeros((N + 1, KB))
    shear[:, :KB - 1] = 0.05 * np.cos(np.pi * (zz1[:, :KB - 1] + 0.1 * _waves(r, xc, yc)[:, None])) * wetc[:, None]
    live = np.ones(KB)
    live[KB - 1] = 0.0
    st.update(ua=ua, va=va, u=ua[:, None] * live + shear, v=va[:, None] * live - 0.5 * shear)
    # stratification: the run's mean profile and the seed's anomalies
    init = c["init"]
    if init["kind"] == "constant":
        tm, sm = np.full((M + 1, KB), float(init["t"])), np.full((M + 1, KB), float(init["s"]))
    else:
        tm = init["t"][0] + (init["t"][1] - init["t"][0]) * (-zz)
        sm = init["s"][0] + (init["s"][1] - init["s"][0]) * (-zz)
    if init.get("t_offset") is not None:
        tm = tm + np.asarray(init["t_offset"])[:, None]
    tm, sm = tm * live, sm * live
    warm = (0.3 * _waves(r, x, y)[:, None] * (1.0 + zz)) * live
    salt = (0.2 * _waves(r, x, y)[:, None] * (1.0 + zz)) * live
    t1, s1 = tm + warm, sm + salt

    def density(t, s):
        rho = dens2(s, t)
        rho[:, KB - 1] = 0.0
        rho[0] = 0.0
        return rho

    rho1, rmean1 = density(t1, s1), density(tm, sm)
    st.update(t1=t1, s1=s1, tf1=t1, sf1=s1, tmean1=tm, smean1=sm, rho1=rho1, rmean1=rmean1,
              rho=_n2e(g, rho1), rmean=_n2e(g, rmean1), t=_n2e(g, t1), s=_n2e(g, s1))
    # turbulence: a few decades above its floor near the surface and the bed
    inner = np.zeros(KB)
    inner[1:KB - 1] = 1.0
    shape = np.exp(-((z + 0.05) / 0.15) ** 2) + 0.5 * np.exp(-((z + 1.0) / 0.15) ** 2)
    q2 = (2.0e-7 + 5.0e-5 * shape * (1.0 + 0.5 * _waves(r, x, y)[:, None])) * inner
    length = 0.05 + 0.1 * (-z) * (1.0 + z)
    km = (2.0e-4 + 0.3 * length * np.sqrt(q2)) * inner
    st.update(q2=q2, q2l=q2 * length, q2f=q2, q2lf=q2 * length, l=length * inner, km=km, kh=km, kq=km,
              km1=_n2e(g, km))
    for k, a in st.items():
        a = np.array(a)
        a[0] = 0
        st[k] = a.reshape(-1, order="F") if a.ndim > 1 else a
    st["iswetce"][0] = st["iswetct"][0] = st["iswetc"][0] = st["iswetn"][0] = st["iswetnt"][0] = 1
    return st


def _model(base, r, precision):
    c, iint, t0 = _forced(base, r)
    model = Fvcom(c, state=_state(c, r, iint, t0))
    model.set_clock(iint, t0)
    model.set_precision(precision)
    return model, c


class _Reader:
    """Output buffers in pinned host memory, filled by fvg_get_field."""

    def __init__(self, model, fields, single):
        lib = model.lib
        lib.fvg_get_field.argtypes = [C.c_void_p, C.c_char_p, C.POINTER(C.c_double), C.c_int64]
        self.model, self.single = model, single
        self.buf = {f: torch.empty(model.size(f), dtype=torch.float64).pin_memory() for f in fields}
        self.out = {f: torch.empty(b.shape, dtype=torch.float32) for f, b in self.buf.items()} if single else self.buf

    def read(self):
        m = self.model
        for f, b in self.buf.items():
            if m.lib.fvg_get_field(m.h, f.encode(), C.cast(b.data_ptr(), C.POINTER(C.c_double)), b.numel()):
                raise RuntimeError("fvg_get_field(%s)" % f)
            if self.single:
                self.out[f].copy_(b)
        return self.out


# --------------------------------------------------------------------------------------
# the network's samples
# --------------------------------------------------------------------------------------
def _samples(n, seed):
    """Standardised inputs, and targets that the network can represent."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((n, 8), generator=gen, device="cuda", dtype=torch.float32)
    y = torch.stack([torch.tanh(x[:, 0] - 0.5 * x[:, 1]), 0.3 * x[:, 2] * x[:, 3],
                     torch.sin(x[:, 4]) + 0.1 * x[:, 7]], dim=1).contiguous()
    return x, y


def _params(n, seed):
    return (0.2 * np.random.default_rng(seed).standard_normal(n)).astype(np.float32)


# --------------------------------------------------------------------------------------
def prepare(case, seed):
    r = np.random.default_rng(seed)
    if case["kind"] in ("train", "forward"):
        net = Mlp(seed=1)
        x, y = _samples(case["n"], seed)
        state = dict(case=case, net=net, x=x, y=y, params=_params(net.npar, seed), seed=seed)
        net.set_params(state["params"])
        if case["kind"] == "forward":
            state["out"] = torch.zeros((case["n"], 3), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        return state
    if case["kind"] == "group":
        coast = _mesh(dict(kind="coast", npts=case["npts"], kb=case["kb"], members=case["members"], option="plain"))
        key = ("channels", case["channels"])
        if key not in _MESH:
            one = _mesh(dict(kind="channel", nx=100, ny=20, kb=11, river="node"))
            _MESH[key] = ensemble.union_case(one, ensemble.perturbed_members(one, case["channels"], seed=6))
        a, _ = _model(coast, r, "fp32flux")
        closure.attach(a, closure.load(CLOSURE))
        b, _ = _model(_MESH[key], r, "fp32flux")
        return dict(case=case, group=Group([a, b]), models=[a, b], read=[_Reader(m, FIELDS, True) for m in (a, b)])
    model, c = _model(_mesh(case), r, case["precision"])
    state = dict(case=case, model=model)
    if case["call"] == "coupled":
        state["read"] = _Reader(model, ("el", "ua", "va"), case["precision"] != "fp64")
        state["wind"] = [torch.from_numpy(np.array(s)).pin_memory() for s in wind_stress(c)]
        model.lib.fvg_set_field.argtypes = [C.c_void_p, C.c_char_p, C.POINTER(C.c_double), C.c_int64]
    else:
        state["read"] = _Reader(model, FIELDS, case["precision"] != "fp64")
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        net = state["net"]
        net.set_params(state["params"])
        history = net.train(state["x"].data_ptr(), state["y"].data_ptr(), case["n"], case["epochs"], case["batch"],
                            2e-3, seed=state["seed"])
        return {"params": net.params(), "history": history}
    if case["kind"] == "forward":
        state["net"].forward(state["x"].data_ptr(), case["n"], state["out"].data_ptr())
        return state["out"]
    if case["kind"] == "group":
        state["group"].run(case["steps"])
        return [rd.read() for rd in state["read"]]
    model = state["model"]
    if case["call"] == "coupled":
        for _ in range(case["steps"]):
            for name, w in zip((b"wstress_x", b"wstress_y"), state["wind"]):
                if model.lib.fvg_set_field(model.h, name, C.cast(w.data_ptr(), C.POINTER(C.c_double)), w.numel()):
                    raise RuntimeError("fvg_set_field")
            model.internal_step()
            out = state["read"].read()
        return out
    model.run(case["steps"])
    return state["read"].read()


def exact(case, seed):
    """The network's outputs in 64 bits.  The time step has no restatement outside this
    repository that would fit here: its outputs are held to their types' bounds."""
    if case["kind"] != "forward":
        return None
    x, _ = _samples(case["n"], seed)
    p = torch.from_numpy(_params(4931, seed)).to("cuda", torch.float64)
    w1, b1, w2, b2, w3, b3 = torch.split(p, (512, 64, 4096, 64, 192, 3))

    def gelu(v):
        return 0.5 * v * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (v + 0.044715 * v ** 3)))

    h = gelu(x.double() @ w1.view(64, 8).T + b1)
    h = gelu(h @ w2.view(64, 64).T + b2)
    return h @ w3.view(3, 64).T + b3


def work(case):
    """One step cannot do without reading and writing its prognostic fields (3-D: U, V on
    cells, T, S, q2, q2l and three mixing coefficients on nodes; 2-D: elevation and mean
    currents), the mesh's lists and metrics once, and the arithmetic of its flux loops (per
    cell, node and layer, and per cell and stage of the external mode)."""
    if case["kind"] == "train":
        return {"bytes": 44.0 * case["n"] * case["epochs"], "flops": 6.0 * 4800 * case["n"] * case["epochs"]}
    if case["kind"] == "forward":
        return {"bytes": 44.0 * case["n"], "flops": 2.0 * 4800 * case["n"]}
    if case["kind"] == "group":
        parts = [(case["npts"] * case["members"], case["kb"] - 1), (2121 * case["channels"], 10)]
    elif case["kind"] == "channel":
        parts = [((case["nx"] + 1) * (case["ny"] + 1), case["kb"] - 1)]
    else:
        parts = [(case["npts"] * case["members"], case["kb"] - 1)]
    total = {"bytes": 0.0, "flops": 0.0}
    for m, k in parts:
        n = 2 * m
        stages = 40 * case["steps"]
        total["bytes"] += case["steps"] * (8.0 * 2 * k * (2 * n + 7 * m) + 200.0 * n + 150.0 * m) + 16.0 * stages * (m + 2 * n)
        total["flops"] += case["steps"] * k * (450.0 * n + 700.0 * m) + stages * (320.0 * n + 90.0 * m)
    return total
