"""The work that a user of this framework has it do, as cases that can be timed.

A pass is what the user's own time loop does: a time step is the CFL maximum
read back, dt on the host and the step replayed as a graph
(``Solver.time_step`` and ``Solver.evolve``), with the rigid-body half steps
around it where bodies move; a batch advances all of its cases; the learned
sensor is trained by one optimisation step.  The node array is uploaded once,
as for any run, and stays on the GPU.

``form`` is the arithmetic form: "fp64" (the drop-in default), "bulk" (FP32
fluxes) and "hybrid" (FP32 fluxes with the learned sensor).  The FP64 form's
fields are returned as they are.  A program that asks for an FP32 form has
asked for FP32 accuracy and takes its fields as float32, which is also what
the reference's data files hold; ``steps`` steps are taken before it does.
``tune`` is true where the program lets the library time its stage kernels
before a long run (acfd_autotune), false where it runs on the defaults, as
short runs and the drop-in program do.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from artracfd_b200 import abi, configs, sensor
from artracfd_b200.batch import Batch
from artracfd_b200.case import Boundary, CaseSpec
from artracfd_b200.solver import Solver

GAMMA = 1.4
FORMS = {"fp64": abi.FP64, "bulk": abi.FP32_BULK, "hybrid": abi.FP32_HYBRID}


def _step(name, flow, mx, my, mz, form, tune, steps=1, weno5=True, rk3=True, roe=True, llf=True):
    return {"name": name, "flow": flow, "mx": mx, "my": my, "mz": mz, "form": form, "tune": tune, "steps": steps,
            "weno5": weno5, "rk3": rk3, "roe": roe, "llf": llf}


def listed():
    return [
        # the smallest run: a 3D Sod tube on the defaults (launches and read-backs)
        _step("sod-128x8x8-fp64", "sod", 128, 8, 8, "fp64", False),
        # a small vortex run in the form with the learned sensor
        _step("tgv-64-hybrid", "tgv", 64, 64, 64, "hybrid", True, steps=2),
        # the headline workload, viscous TGV 128^3, in the forms it is run in
        _step("tgv-128-fp64", "tgv", 128, 128, 128, "fp64", True),
        _step("tgv-128-bulk", "tgv", 128, 128, 128, "bulk", True, steps=2),
        _step("tgv-128-hybrid", "tgv", 128, 128, 128, "hybrid", True, steps=2),
        # ragged extents, discontinuities and outflow faces: a viscous 3D Riemann problem
        _step("riemann-159x97x61-bulk", "riemann", 159, 97, 61, "bulk", True, steps=2),
        # walls and inflow, the scheme's other options (WENO3, RK2, arithmetic mean), defaults
        _step("channel-95x63x33-weno3", "channel", 95, 63, 33, "fp64", False, weno5=False, rk3=False, roe=False),
        # a planar shock over a body in a thin periodic slab, in both forms
        _step("shock-1024x512x4-fp64", "shock", 1024, 512, 4, "fp64", True),
        _step("shock-1024x512x4-hybrid", "shock", 1024, 512, 4, "hybrid", True, steps=2),
        # crossflow over eight moving spheres as the drop-in program runs it (defaults, two
        # rigid-body half steps around the fluid step): the largest
        _step("spheres-192-fp64", "spheres", 192, 192, 192, "fp64", False),
        # a parameter sweep: independent TGV and Riemann cases advanced together
        {"name": "batch-10-hybrid", "flow": "batch", "count": 10, "small": 64, "large": 112, "form": "hybrid",
         "steps": 1},
        # training the sensor: one optimisation step of a batch (forward, backward, Adam)
        {"name": "sensor-train-16384", "flow": "train", "samples": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    flow = rng.choice(["sod", "tgv", "tgv", "riemann", "riemann", "channel", "shock", "spheres", "batch", "train"])
    if flow == "train":
        return {"flow": "train", "samples": _log(rng, 2000, 70000)}
    if flow == "batch":
        lo = rng.randint(24, 70)
        return {"flow": "batch", "count": rng.randint(2, 9), "small": lo, "large": lo + rng.randint(0, 40),
                "form": rng.choice(["bulk", "hybrid"]), "steps": 1}
    form = rng.choice(["fp64", "bulk", "hybrid"])
    if flow == "sod":
        m = (_log(rng, 40, 500), rng.randint(5, 40), rng.randint(5, 40))
    elif flow == "shock":
        m = (_log(rng, 150, 1000), _log(rng, 90, 500), rng.randint(4, 9))
    elif flow == "spheres":
        m = (_log(rng, 60, 130),) * 3
        form = "fp64"
    else:
        m = tuple(_log(rng, 24, 145) for _ in range(3))
    return {"flow": flow, "mx": m[0], "my": m[1], "mz": m[2], "form": form, "tune": flow != "spheres" and
            rng.random() < 0.6, "steps": 1 if form == "fp64" else 2, "weno5": form == "hybrid" or rng.random() < 0.75,
            "rk3": rng.random() < 0.75, "roe": rng.random() < 0.75, "llf": rng.random() < 0.75}


# ----------------------------------------------------------------------
# the flows
# ----------------------------------------------------------------------
def _ref_state(Ma, Re, length=1.0):
    """(refT, refMu, p0) of rho0 = 1, T0 = 1 at Mach number Ma and Reynolds number Re."""
    refT = 1.0 / (Ma * Ma * GAMMA * configs.GAS_R)
    return refT, (length / Re) / configs.sutherland(refT), 1.0 / (GAMMA * Ma * Ma)


def _spec(case, rng):
    """The case description; everything but the initial field."""
    P, O = Boundary(abi.PERIODIC), Boundary(abi.OUTFLOW)
    kw = dict(m=(case["mx"], case["my"], case["mz"]), end=1.0e6, tScheme=int(case["rk3"]), sScheme=int(case["weno5"]),
              jacobMean=int(case["roe"]), fluxSplit=int(not case["llf"]), cfl=0.5)
    flow, tau = case["flow"], 2.0 * math.pi
    if flow == "sod":
        kw.update(domain_lo=(0, 0, 0), domain_hi=(1, 0.0625, 0.0625), cfl=0.6, boundaries=[O, O, P, P, P, P])
    elif flow == "tgv":
        refT, refMu, _ = _ref_state(0.1, 1600.0)
        kw.update(domain_lo=(0, 0, 0), domain_hi=(tau, tau, tau), refT=refT, refMu=refMu, boundaries=[P] * 6)
    elif flow == "riemann":
        refT, refMu, _ = _ref_state(0.3, 1600.0)
        kw.update(domain_lo=(0, 0, 0), domain_hi=(1, 1, 1), refT=refT, refMu=refMu, boundaries=[O] * 6)
    elif flow == "channel":
        refT, refMu, p0 = _ref_state(0.3, 400.0)
        kw.update(domain_lo=(0, 0, 0), domain_hi=(2, 1, 0.5), refT=refT, refMu=refMu,
                  boundaries=[Boundary(abi.INFLOW, (1.0, 0.6, 0.0, 0.0, p0)), O, Boundary(abi.NOSLIPWALL, (1.05,)),
                              Boundary(abi.SLIPWALL, (-1.0,)), P, P])
    elif flow == "shock":
        W = Boundary(abi.SLIPWALL, (-1.0,))
        kw.update(domain_lo=(0, 0, 0), domain_hi=(16, 8, 0.0625),
                  boundaries=[Boundary(abi.INFLOW, configs.POST_SHOCK), O, W, W, P, P])
    elif flow == "spheres":
        refT, refMu, p0 = _ref_state(0.3, 200.0, 0.3)
        kw.update(domain_lo=(0, 0, 0), domain_hi=(4, 4, 4), refT=refT, refMu=refMu, psi=2,
                  boundaries=[Boundary(abi.INFLOW, (1.0, 1.0, 0.0, 0.0, p0)), O, P, P, P, P])
    else:
        raise ValueError(flow)
    return CaseSpec(**kw)


def _waves(rng, x, y, z, extent, amplitude):
    """A few long waves of random phase and direction, periodic over the extents."""
    out = 0.0
    for _ in range(3):
        k = 2.0 * math.pi * rng.integers(-2, 3, size=3) / np.asarray(extent, dtype=np.float64)
        out = out + amplitude / 3.0 * torch.sin(float(k[0]) * x + float(k[1]) * y + float(k[2]) * z +
                                                float(rng.uniform(0.0, 2.0 * math.pi)))
    return out


def _field(flow, lo, hi, x, y, z, rng):
    """rho, u, v, w, p at the given coordinates, made from rng alone."""
    ext = [b - a for a, b in zip(lo, hi)]
    one = torch.ones_like(x + y + z)
    if flow == "tgv":
        p0 = _ref_state(0.1, 1600.0)[2]
        u = torch.sin(x) * torch.cos(y) * torch.cos(z) + _waves(rng, x, y, z, ext, 0.05)
        v = -torch.cos(x) * torch.sin(y) * torch.cos(z) + _waves(rng, x, y, z, ext, 0.05)
        w = _waves(rng, x, y, z, ext, 0.05) * one
        p = p0 + (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2) / 16
        return [one, u * one, v * one, w, p * one]
    if flow == "sod":
        a, b = [1.0, 0.0, 0.0, 0.0, 1.0], [0.125, 0.0, 0.0, 0.0, 0.1]
        at = rng.uniform(0.4, 0.6)
        s = rng.uniform(0.95, 1.05, size=(2, 5))
        return [torch.where(x < at, a[v] * s[0, v], b[v] * s[1, v]) * one for v in range(5)]
    if flow == "riemann":
        p0 = _ref_state(0.3, 1600.0)[2]
        c = rng.uniform(0.4, 0.6, size=3)
        part = ((x > c[0]).long() + 2 * (y > c[1]).long() + 4 * (z > c[2]).long()) * one.long()
        st = np.concatenate([rng.uniform(0.5, 2.0, (8, 1)), rng.uniform(-0.5, 0.5, (8, 3)),
                             p0 * rng.uniform(0.5, 2.0, (8, 1))], axis=1)
        return [torch.as_tensor(st[:, v], device=x.device)[part] for v in range(5)]
    if flow == "channel":
        p0 = _ref_state(0.3, 400.0)[2]
        return [one * (1 + _waves(rng, x, y, z, ext, 0.02)), 0.6 + _waves(rng, x, y, z, ext, 0.1) * one,
                _waves(rng, x, y, z, ext, 0.05) * one, _waves(rng, x, y, z, ext, 0.05) * one,
                p0 * (1 + _waves(rng, x, y, z, ext, 0.02)) * one]
    if flow == "shock":
        at = rng.uniform(1.9, 2.1)
        post = configs.POST_SHOCK
        pre = [1 + _waves(rng, x, y, z, ext, 0.02), 0 * x, 0 * x, 0 * x, 1 + 0 * x]
        return [torch.where(x < at, one * post[v], pre[v] * one) for v in range(5)]
    if flow == "spheres":
        p0 = _ref_state(0.3, 200.0, 0.3)[2]
        return [one * (1 + _waves(rng, x, y, z, ext, 0.02)), one + _waves(rng, x, y, z, ext, 0.02),
                _waves(rng, x, y, z, ext, 0.02) * one, _waves(rng, x, y, z, ext, 0.02) * one, p0 * one]
    raise ValueError(flow)


def _conservative(prim):
    rho, u, v, w, p = prim
    return torch.stack([rho, rho * u, rho * v, rho * w, 0.5 * rho * (u * u + v * v + w * w) + p / (GAMMA - 1.0)])


def _nodes(flow, spec, part, rng):
    """The initial node array (the reference's records): the field on the
    computed nodes, zero flags there and -1 elsewhere."""
    n = [int(v) for v in part.n]
    r = [(int(part.ns[0][s][0]), int(part.ns[0][s][1])) for s in range(3)]
    c = [spec.domain_lo[s] + (torch.arange(*r[s], device="cuda", dtype=torch.float64) - part.ng[s]) * part.d[s]
         for s in range(3)]
    U = _conservative(_field(flow, spec.domain_lo, spec.domain_hi, c[0][None, None, :], c[1][None, :, None],
                             c[2][:, None, None], rng))
    rec = torch.zeros((n[2], n[1], n[0], 17), dtype=torch.float64, device="cuda")
    rec[..., 2:] = 1.0
    inner = rec[r[2][0]:r[2][1], r[1][0]:r[1][1], r[0][0]:r[0][1]]
    inner[..., 2:7] = U.permute(1, 2, 3, 0)
    rec.view(torch.int32)[..., :4] = -1
    inner.view(torch.int32)[..., :4] = 0
    return rec.cpu().numpy().reshape(-1).view(abi.NODE_DTYPE)


def _sphere(centre, radius, velocity):
    P = abi.Polyhedron()
    P.faceN, P.edgeN, P.vertN = 0, 0, 0
    P.state = 0 if velocity is not None else 1
    P.r = radius
    P.T, P.cf, P.area = -1.0, 1.0 if velocity is not None else 0.0, 4.0 * math.pi * radius * radius
    for s in range(3):
        P.O[s] = float(centre[s])
        P.V[s] = float(velocity[s]) if velocity is not None else 0.0
        P.box[s][0], P.box[s][1] = P.O[s] - radius, P.O[s] + radius
    return P


def _bodies(flow, seed):
    if flow == "spheres":
        centres, vel = configs.sphere_centres(8, seed=seed)
        return [_sphere(c, 0.15, v) for c, v in zip(centres, vel)]
    if flow == "shock":
        return [_sphere((4.0, 4.0, 0.03125), 0.5, None)]
    return []


_STREAMS = []


def _stream():
    """The one stream that the program's work goes to."""
    if not _STREAMS:
        _STREAMS.append(torch.cuda.Stream())
    return _STREAMS[0]


class _Memory:
    """Device memory of the library as torch sees it; it keeps its owner alive."""

    def __init__(self, owner, ptr, shape, strides, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "strides": strides, "typestr": kind,
                                         "version": 3}


def _state_view(solver, owner):
    """U[TO] of every node as a tensor [variable, z, y, x] over the library's
    memory, and the node types did [z, y, x]."""
    ptr, flags, pitch, plane = solver.device_state()
    n = solver.part.n
    U = torch.as_tensor(_Memory(owner, ptr, (5, n[2], n[1], n[0]), (plane * 8, pitch * n[1] * 8, pitch * 8, 8),
                                "<f8"), device="cuda")
    did = torch.as_tensor(_Memory(owner, flags, (n[2], n[1], n[0]), (pitch * n[1] * 4, pitch * 4, 4), "<i4"),
                          device="cuda")
    return U, did


# ----------------------------------------------------------------------
# what a program has in hand, and a pass
# ----------------------------------------------------------------------
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    flow = case["flow"]
    if flow == "train":
        return _prepare_train(case, rng)
    if flow == "batch":
        return _prepare_batch(case, rng)
    spec = _spec(case, rng)
    part, model = spec.descriptors()
    node = _nodes(flow, spec, part, rng)
    hybrid = case["form"] == "hybrid"
    s = Solver(part, model, abi.FP64 if hybrid else FORMS[case["form"]])
    s.set_stream(_stream().cuda_stream)
    if hybrid:
        sensor.attach(s)
    s.upload(node)
    geo = _bodies(flow, seed)
    if geo:
        s.geo_upload(geo)
        s.compute_geometric_field()
    s.treat_boundary(abi.TO)
    if case["tune"]:
        s.autotune()
    U, did = _state_view(s, s)
    torch.cuda.synchronize()
    return {"case": case, "solver": s, "cfl": spec.cfl, "U": U, "did": did}


def _batch_specs(case):
    """(flow, description) of the batch's cases: vortices and Riemann problems in turn."""
    out = []
    for q, n in enumerate(np.linspace(case["small"], case["large"], case["count"])):
        Re = 400.0 * (1 + q % 8)
        out.append(("tgv", configs.tgv(n=int(n), Re=Re, Ma=0.1, stepN=0)) if q % 2 == 0 else
                   ("riemann", configs.riemann_viscous(n=int(n), Re=Re, Ma=0.3, rng=np.random.default_rng(q))))
    return out


def _prepare_batch(case, rng):
    flows, specs = zip(*_batch_specs(case))
    b = Batch([s.descriptors() for s in specs])
    for c, spec in enumerate(specs):
        b.upload(c, _nodes(flows[c], spec, b.parts[c], rng))
        b.treat_boundary(c)
    if case["form"] == "hybrid":
        params, threshold, _ = sensor.load()
        b.sensor_load(params, threshold)
    b.set_precision(FORMS[case["form"]])
    b.set_stream(_stream().cuda_stream)
    torch.cuda.synchronize()
    return {"case": case, "batch": b, "cfl": [s.cfl for s in specs],
            "U": [_state_view(v, b)[0] for v in b.views]}


def _prepare_train(case, rng):
    n = case["samples"]
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 31)))
    # stencils of smooth and jumping densities and pressures, as the sensor's features:
    # ten times the deviation from the stencil mean over the mean
    q = 1.0 + 0.02 * torch.randn((n, 2, 5), device="cuda", generator=g)
    jump = (torch.rand((n, 1, 1), device="cuda", generator=g) < 0.2) * torch.rand((n, 2, 1), device="cuda", generator=g)
    q = q + jump * (torch.arange(5, device="cuda") > 2)
    mean = q.mean(dim=2, keepdim=True)
    X = (10.0 * (q / mean - 1.0)).reshape(n, 10).float().contiguous()
    y = ((q.amax(dim=2) - q.amin(dim=2)).amax(dim=1) > 0.15).float().contiguous()
    lib = abi.load_library()
    params = torch.tensor(sensor.init_params(int(rng.integers(1 << 31))), device="cuda")
    zero = torch.zeros_like(params)
    return {"case": case, "lib": lib, "X": X, "y": y, "params": params, "grad": zero.clone(), "m": zero.clone(),
            "v": zero.clone(), "loss": torch.zeros(1, device="cuda"), "step": 0}


def run(state):
    flow = state["case"]["flow"]
    if flow == "train":
        return _run_train(state)
    if flow == "batch":
        dts = state["batch"].advance(state["cfl"], state["case"]["steps"])
        with torch.cuda.stream(_stream()):
            return {"U": [u.float() for u in state["U"]], "dt": dts.astype(np.float32)}
    s, dt = state["solver"], 0.0
    for _ in range(state["case"]["steps"]):
        dt = s.time_step(state["cfl"])
        if flow == "spheres":
            _solid_half_step(s, 0.5 * dt)
        s.evolve(dt, graph=True)
        if flow == "spheres":
            _solid_half_step(s, 0.5 * dt)
    with torch.cuda.stream(_stream()):
        out = {"U": state["U"] if state["case"]["form"] == "fp64" else state["U"].float(), "dt": dt}
    if s.geo:
        out["did"] = state["did"]
    return out


def _solid_half_step(s, dt):
    """The rigid-body half step with prescribed velocities: surface forces and
    contacts read back, the bodies moved, the nodes mapped anew."""
    s.integrate_surface_force()
    s.collision_scan()
    for P in s.geo:
        for d in range(3):
            P.O[d] += P.V[d] * dt
            P.box[d][0], P.box[d][1] = P.O[d] - P.r, P.O[d] + P.r
    s.geo_upload(s.geo)
    s.compute_geometric_field()
    s.treat_ib(abi.TO)


def _run_train(st):
    lib, vp = st["lib"], ctypes.c_void_p
    stream = vp(torch.cuda.current_stream().cuda_stream)
    st["grad"].zero_()
    st["loss"].zero_()
    st["step"] += 1
    n = st["X"].shape[0]
    abi.check(lib.acfd_mlp_grad(vp(st["params"].data_ptr()), vp(st["X"].data_ptr()), vp(st["y"].data_ptr()), n, 3.0,
                                vp(st["grad"].data_ptr()), vp(st["loss"].data_ptr()), stream), lib)
    abi.check(lib.acfd_mlp_adam(vp(st["params"].data_ptr()), vp(st["grad"].data_ptr()), vp(st["m"].data_ptr()),
                                vp(st["v"].data_ptr()), st["step"], 1e-3, 1.0 / n, stream), lib)
    return {"grad": st["grad"], "loss": st["loss"], "m": st["m"]}


# ----------------------------------------------------------------------
# the work of a pass
# ----------------------------------------------------------------------
def _step_work(m, viscous, rk3, steps):
    """Every computed node's state read and written once a step; the scheme's
    own operations a node and stage (characteristic WENO flux, viscous flux
    and update: 1,535, without the viscous part 1,420) of the six half steps."""
    nodes = float((m[0] + 1) * (m[1] + 1) * (m[2] + 1))
    flops = (1535.0 if viscous else 1420.0) * 6 * (3 if rk3 else 2)
    return {"bytes": 80.0 * nodes * steps, "flops": flops * nodes * steps}


def work(case):
    flow = case["flow"]
    if flow == "train":
        n = float(case["samples"])
        return {"bytes": 44.0 * n + 6 * 4 * 1441.0, "flops": 6.0 * (10 * 32 + 32 * 32 + 32) * n}
    if flow == "batch":
        all_ = [_step_work((int(n),) * 3, True, True, case["steps"])
                for n in np.linspace(case["small"], case["large"], case["count"])]
        return {k: sum(w[k] for w in all_) for k in ("bytes", "flops")}
    w = _step_work((case["mx"], case["my"], case["mz"]), flow not in ("sod", "shock"), case["rk3"], case["steps"])
    return {"bytes": w["bytes"], "flops": w["flops"] * (1.0 if case["weno5"] else 0.55)}


# ----------------------------------------------------------------------
# the same values in 64 bits
# ----------------------------------------------------------------------
class _Exact:
    """The scheme on plain float64 tensors [variable, z, y, x]: WENO on the
    Roe-averaged (or arithmetic) characteristic split fluxes, central viscous
    fluxes, RK stages inside the split half steps Z, Y, X, X, Y, Z, ghost
    layers filled face by face."""

    def __init__(self, spec, weno5, rk3, roe, llf):
        self.weno5, self.rk3, self.roe, self.llf = weno5, rk3, roe, llf
        self.kind = [b.kind for b in spec.boundaries]
        self.values = [b.values for b in spec.boundaries]
        gl = 3 if weno5 else 2
        self.m = [int(v) for v in spec.m]
        per = [self.kind[2 * s] == abi.PERIODIC for s in range(3)]
        self.ng = [gl if p else gl - 1 for p in per]
        self.n = [self.m[s] + 1 + 2 * self.ng[s] for s in range(3)]
        self.lo = [self.ng[s] + (not per[s]) for s in range(3)]
        self.hi = [self.n[s] - self.ng[s] - (not per[s]) for s in range(3)]
        self.d = [(spec.domain_hi[s] - spec.domain_lo[s]) / self.m[s] for s in range(3)]
        self.gas = configs.GAS_R * spec.refT  # 1 / (gamma Ma^2) of the reference velocity 1
        self.cv = self.gas / (GAMMA - 1.0)
        self.mu, self.refT = spec.refMu, spec.refT
        c = [spec.domain_lo[s] + (torch.arange(self.lo[s], self.hi[s], device="cuda", dtype=torch.float64) - self.ng[s])
             * self.d[s] for s in range(3)]
        self.c = [c[0][None, None, :], c[1][None, :, None], c[2][:, None, None]]

    def box(self, U, shift=(0, 0, 0), grow=None):
        lo, hi = list(self.lo), list(self.hi)
        if grow is not None:
            lo[grow] -= 1
        return U[:, lo[2] + shift[2]:hi[2] + shift[2], lo[1] + shift[1]:hi[1] + shift[1],
                 lo[0] + shift[0]:hi[0] + shift[0]]

    def prim(self, U):
        p = (U[4] - 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2) / U[0]) * (GAMMA - 1.0)
        return torch.stack([U[0], U[1] / U[0], U[2] / U[0], U[3] / U[0], p, p / (U[0] * self.gas)])

    def cons(self, V, p, T):
        rho = p / (T * self.gas)
        return _conservative([rho, V[0], V[1], V[2], p])

    def fill(self, U):
        for r in range(max(self.ng) + 1):
            for face in range(6):
                s, sign = face // 2, -1 if face % 2 == 0 else 1
                kind = self.kind[face]
                if r > self.ng[s] or (r == 0 and kind == abi.PERIODIC):
                    continue
                a, b = [], []
                for t in range(3):
                    w = min(r, self.ng[t])
                    if t == s:
                        first = self.ng[t] - r if sign < 0 else self.n[t] - self.ng[t] - 1 + r
                        a.append(first)
                        b.append(first + 1)
                    else:
                        a.append(self.ng[t] - w)
                        b.append(self.n[t] - self.ng[t] + w)

                def at(k):
                    q = [(a[t], b[t]) if t != s else (a[t] - k * sign, b[t] - k * sign) for t in range(3)]
                    return U[:, q[2][0]:q[2][1], q[1][0]:q[1][1], q[0][0]:q[0][1]]

                if kind == abi.PERIODIC:
                    new = at(self.m[s])
                elif kind in (abi.SLIPWALL, abi.NOSLIPWALL):
                    if r == 0:
                        h = self.prim(at(1))
                        V = h[1:4].clone()
                        if kind == abi.SLIPWALL:
                            V[s] = 0.0
                        else:
                            V[:] = 0.0
                        given = self.values[face][0] if self.values[face] else -1.0
                        new = self.cons(V, h[4], h[5] if given < 0.0 else torch.full_like(h[5], given))
                    else:
                        o, i = self.prim(at(r)), self.prim(at(2 * r))
                        new = self.cons(2.0 * o[1:4] - i[1:4], i[4], i[5])
                elif kind == abi.INFLOW and r == 0:
                    rho, u, v, w, p = self.values[face][:5]
                    given = torch.tensor([rho, rho * u, rho * v, rho * w,
                                          0.5 * rho * (u * u + v * v + w * w) + p / (GAMMA - 1.0)],
                                         dtype=torch.float64, device="cuda")
                    new = given[:, None, None, None]
                else:
                    new = at(1)
                at(0)[...] = new.clone()

    def dt(self, U, cfl):
        q = self.prim(self.box(U))
        c = torch.sqrt(GAMMA * self.gas * q[5])
        return cfl * min(self.d[s] / float((q[1 + s].abs() + c).max()) for s in range(3))

    def weno(self, f):
        eps = 1.0e-6
        if self.weno5:
            b = [13.0 / 12.0 * (f[0] - 2 * f[1] + f[2]) ** 2 + 0.25 * (f[0] - 4 * f[1] + 3 * f[2]) ** 2,
                 13.0 / 12.0 * (f[1] - 2 * f[2] + f[3]) ** 2 + 0.25 * (f[1] - f[3]) ** 2,
                 13.0 / 12.0 * (f[2] - 2 * f[3] + f[4]) ** 2 + 0.25 * (3 * f[2] - 4 * f[3] + f[4]) ** 2]
            q = [(2 * f[0] - 7 * f[1] + 11 * f[2]) / 6, (-f[1] + 5 * f[2] + 2 * f[3]) / 6,
                 (2 * f[2] + 5 * f[3] - f[4]) / 6]
            g = [0.1, 0.6, 0.3]
        else:
            b = [(f[1] - f[0]) ** 2, (f[2] - f[1]) ** 2]
            q = [(-f[0] + 3 * f[1]) / 2, (f[1] + f[2]) / 2]
            g = [1.0 / 3.0, 2.0 / 3.0]
        w = [gk / (eps + bk) ** 2 for gk, bk in zip(g, b)]
        return sum(wk * qk for wk, qk in zip(w, q)) / sum(w)

    def flux(self, U, s):
        """The flux at the interfaces lo-1/2 .. hi-1/2 of axis s."""
        h = 3 if self.weno5 else 2
        e = [0, 0, 0]

        def node(k):
            sh = list(e)
            sh[s] = k
            return self.box(U, sh, grow=s)

        St = [node(k) for k in range(1 - h, h + 1)]  # around the interface right of node 0
        L, R = St[h - 1], St[h]

        def side(u):
            V = u[1:4] / u[0]
            return V, u[4] / u[0] * GAMMA - 0.5 * (V ** 2).sum(0) * (GAMMA - 1.0)

        (VL, HL), (VR, HR) = side(L), side(R)
        D = torch.sqrt(R[0] / L[0]) if self.roe else torch.ones_like(L[0])
        V, H = (VL + D * VR) / (1 + D), (HL + D * HR) / (1 + D)
        q = 0.5 * (V ** 2).sum(0)
        c = torch.sqrt((GAMMA - 1.0) * (H - q))
        lam = [V[s] - c, V[s], V[s], V[s], V[s] + c]
        big = [V[s].abs() + c] * 5 if self.llf else [torch.sqrt(l * l + 1.0e-6) for l in lam]
        b, d = (GAMMA - 1.0) / (2 * c * c), 1.0 / (2 * c)
        Wc = []
        for u in St:
            A = q * u[0] - (V * u[1:4]).sum(0) + u[4]
            B = V[s] * u[0] - u[1 + s]
            mid = [u[0] - 2 * b * A if t == s else u[1 + t] - 2 * b * V[t] * A for t in range(3)]
            Wc.append([b * A + d * B] + mid + [b * A - d * B])
        G = []
        for r in range(5):
            lp, ln = 0.5 * (lam[r] + big[r]), 0.5 * (lam[r] - big[r])
            k = 2 * h - 1
            G.append(self.weno([lp * Wc[i][r] for i in range(k)]) +
                     self.weno([ln * Wc[2 * h - 1 - i][r] for i in range(k)]))
        a, z = G[0] + G[4], G[4] - G[0]
        F = [a + G[1 + s]]
        F += [V[t] * (a + G[1 + s]) + c * z if t == s else V[t] * a + G[1 + t] for t in range(3)]
        F.append(H * a + V[s] * c * z + (V[s] ** 2 - q) * G[1 + s] + sum(V[t] * G[1 + t] for t in range(3) if t != s))
        F = torch.stack(F)
        if self.mu > 0.0:
            F = F - self.viscous(U, s)
        return F

    def viscous(self, U, s):
        def node(t, k, j):
            sh = [0, 0, 0]
            sh[s] += j
            if t is not None:
                sh[t] += k
            u = self.box(U, sh, grow=s)
            return u

        def vel(u):
            return u[1:4] / u[0]

        def temp(u):
            return (u[4] - 0.5 * (u[1] ** 2 + u[2] ** 2 + u[3] ** 2) / u[0]) / (u[0] * self.cv)

        c, p = node(None, 0, 0), node(None, 0, 1)
        Vc, Vp, Tc, Tp = vel(c), vel(p), temp(c), temp(p)
        g = [None] * 3  # g[t][a] = d v_a / d x_t
        g[s] = (Vp - Vc) / self.d[s]
        for t in range(3):
            if t != s:
                ahead, behind = vel(node(t, 1, 0)) + vel(node(t, 1, 1)), vel(node(t, -1, 0)) + vel(node(t, -1, 1))
                g[t] = 0.25 * (ahead - behind) / self.d[t]
        T = 0.5 * (Tc + Tp) * self.refT
        mu = self.mu * 1.458e-6 * T ** 1.5 / (T + 110.4)
        div = g[0][0] + g[1][1] + g[2][2]
        tau = [mu * (2 * g[s][s] - 2.0 / 3.0 * div) if t == s else mu * (g[t][s] + g[s][t]) for t in range(3)]
        Vh = 0.5 * (Vc + Vp)
        heat = GAMMA * self.cv / 0.71 * mu * (Tp - Tc) / self.d[s]
        return torch.stack([torch.zeros_like(heat)] + tau + [heat + sum(tau[t] * Vh[t] for t in range(3))])

    def stage(self, U, dt, s):
        F = self.flux(U, s)
        ax = 3 - s
        k = F.shape[ax]
        return self.box(U) + dt / self.d[s] * (F.narrow(ax, 0, k - 1) - F.narrow(ax, 1, k - 1))

    def step(self, U, dt):
        for s in (2, 1, 0, 0, 1, 2):
            h, U0 = 0.5 * dt, self.box(U).clone()
            coef = [(0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)] if self.rk3 else [(0.0, 1.0), (0.5, 0.5)]
            for a, b in coef:
                new = a * U0 + b * self.stage(U, h, s)
                self.box(U)[...] = new
                self.fill(U)
        return U


def _exact_run(spec, flow, rng, steps, weno5=True, rk3=True, roe=True, llf=True):
    E = _Exact(spec, weno5, rk3, roe, llf)
    U = torch.ones((5, E.n[2], E.n[1], E.n[0]), dtype=torch.float64, device="cuda")
    E.box(U)[...] = _conservative(_field(flow, spec.domain_lo, spec.domain_hi, *E.c, rng))
    E.fill(U)
    dt = 0.0
    for _ in range(steps):
        dt = E.dt(U, spec.cfl)
        U = E.step(U, dt)
    return U, dt


def exact(case, seed):
    rng = np.random.default_rng(seed)
    flow = case["flow"]
    if flow in ("shock", "spheres"):
        return None  # immersed bodies: their ghost values have no short plain form
    if flow == "train":
        return _exact_train(case, rng)
    if flow == "batch":
        got = [_exact_run(spec, f, rng, case["steps"]) for f, spec in _batch_specs(case)]
        return {"U": [U for U, _ in got], "dt": np.array([[dt for _, dt in got]])}
    spec = _spec(case, rng)
    U, dt = _exact_run(spec, flow, rng, case["steps"], case["weno5"], case["rk3"], case["roe"], case["llf"])
    return {"U": U, "dt": dt}


def _exact_train(case, rng):
    st = _prepare_train(case, rng)
    p = st["params"].double().requires_grad_(True)
    X, y = st["X"].double(), st["y"].double()
    o = np.cumsum([0, 320, 32, 1024, 32, 32, 1])
    W1, b1, W2, b2, w3, b3 = (p[o[i]:o[i + 1]] for i in range(6))
    h = torch.relu(X @ W1.reshape(32, 10).T + b1)
    h = torch.relu(h @ W2.reshape(32, 32).T + b2)
    z = h @ w3 + b3
    w = torch.where(y > 0.5, 3.0, 1.0).double()
    loss = (w * (torch.nn.functional.softplus(z) - y * z)).sum()
    loss.backward()
    return {"grad": p.grad, "loss": loss.detach().reshape(1), "m": 0.1 * p.grad / X.shape[0]}
