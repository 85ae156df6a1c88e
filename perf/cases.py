"""The workloads whose speed is tracked, through the calls a user's program makes.

Three ways into the framework: the resident ``Lattice`` (set_state, step or
step_graph, read), a ``Batch`` of lattices advanced together, and the drop-in
``lattice_boltzmann_step`` on device tensors or on NumPy arrays.  The sizes are
those of the reference's experiments and of the benchmark configurations (shear
wave 64x64, Poiseuille 200x60, von Karman 420x180, cavities 1024^2 ... 8192^2,
the ragged channel sweep); ``draw`` spreads over the whole range between and
beside them.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from lattice_boltzmann_parallel_solver_gb300 import Lattice
from lattice_boltzmann_parallel_solver_gb300 import boundary_utils as BU
from lattice_boltzmann_parallel_solver_gb300 import lattice_boltzmann_method as LBM
from lattice_boltzmann_parallel_solver_gb300.batch import Batch, Member

# wall, lid, inlet speeds and the pressure difference of the experiments
U_WALL, U_LID, U_IN, DELTA_RHO = 0.05, 0.1, 0.1, 1e-3

CX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 1, 1, -1, -1)
OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
W = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4


def _resident(name, kind, nx, ny, storage, omega, steps, graph=False, probe=False):
    return {"name": name, "path": "resident", "kind": kind, "nx": nx, "ny": ny, "storage": storage,
            "omega": omega, "steps": steps, "graph": graph, "probe": probe}


def _batch(name, members, nx_lo, nx_hi, aspect_lo, aspect_hi, storage, steps, layout, graph=False, probe=False):
    return {"name": name, "path": "batch", "members": members, "nx_lo": nx_lo, "nx_hi": nx_hi,
            "aspect_lo": aspect_lo, "aspect_hi": aspect_hi, "storage": storage, "steps": steps, "layout": layout,
            "graph": graph, "probe": probe}


def _step(name, where, kind, nx, ny, omega):
    return {"name": name, "path": where, "kind": kind, "nx": nx, "ny": ny, "omega": omega}


def listed():
    return [
        # the shear-wave decay experiment: a lattice so small that each step is all latency
        _resident("shear_64_fx64", "periodic", 64, 64, "fx64", 1.0, 2000),
        # the Poiseuille experiment (pressure rewrite), replayed from a captured graph
        _resident("poiseuille_200x60_fx64", "poiseuille", 200, 60, "fx64", 1.0, 2000, graph=True),
        # the von Karman channel with its per-step probe, in the default storage ...
        _resident("channel_420x180_fx64", "channel", 420, 180, "fx64", 1.0 / 0.62, 1000, probe=True),
        # ... and in the reduced precision of the precision study
        _resident("channel_420x180_f16", "channel", 420, 180, "f16", 1.0 / 0.62, 1000, probe=True),
        # the cavity bandwidth benchmark: plain FP64, FP32, 16-bit storage, and its largest size in the default storage
        _resident("cavity_1024_f64", "cavity", 1024, 1024, "f64", 1.7, 100),
        _resident("cavity_1024_f32", "cavity", 1024, 1024, "f32", 1.7, 200),
        _resident("cavity_4096_f16", "cavity", 4096, 4096, "f16", 1.7, 200),
        _resident("cavity_8192_fx64", "cavity", 8192, 8192, "fx64", 1.7, 100),
        # the Reynolds-number sweep: a handful of equal channels with probes as one graph-replayed batch
        _batch("reynolds_sweep_fx64", 6, 420, 420, 3 / 7, 3 / 7, "fx64", 1000, 0, graph=True, probe=True),
        # the batched design sweep: many channels of uneven, ragged sizes
        _batch("design_sweep_f16", 20, 200, 1200, 0.3, 0.5, "f16", 100, 1),
        # the drop-in step a driver's loop calls: arrays on the device, and NumPy arrays in and out
        _step("device_step_420x180", "device_step", "channel", 420, 180, 1.0 / 0.62),
        _step("host_step_1024", "host_step", "cavity", 1024, 1024, 1.7),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    case = _draw(rng)
    del case["name"]
    return case


def _draw(rng):
    path = rng.choice(["resident"] * 5 + ["batch", "batch", "device_step", "host_step"])
    if path == "batch":
        few = rng.random() < 0.4
        if few:  # experiment sweeps: a few channels of the experiments' sizes
            storage = rng.choice(["fx64", "fx64", "f64", "f32", "f16"])
            lo = rng.randint(200, 500)
            return _batch(None, rng.randint(3, 10), lo, lo + rng.randint(0, 600), 0.2, 0.6, storage,
                          rng.randint(200, 800), rng.randrange(1 << 30), rng.random() < 0.5, rng.random() < 0.5)
        storage = rng.choice(["f16", "f16", "bf16", "f32", "fx64"])
        return _batch(None, rng.randint(8, 16), 200, rng.randint(400, 1200), 0.3, 0.5, storage, rng.randint(40, 100),
                      rng.randrange(1 << 30), False, rng.random() < 0.3)
    kind = rng.choice(["periodic", "couette", "poiseuille", "channel", "cavity"])
    omega = rng.uniform(0.7, 1.6)
    most = {"resident": 1 << 24, "device_step": 1 << 22, "host_step": 1 << 20}[path]
    nodes = _log_int(rng, 600, most)
    aspect = math.exp(rng.uniform(math.log(0.5), math.log(4.0)))
    nx = max(20, int(round(math.sqrt(nodes * aspect))))
    ny = max(20, int(round(nodes / nx)))
    if path != "resident":
        return _step(None, path, kind, nx, ny, omega)
    storage = rng.choice(["fx64", "fx64", "fx64", "f64", "f32", "f32", "f16", "f16", "bf16"])
    # at most 2^28 node updates: below the largest listed case's time in the slowest storage too
    most_steps = max(20, min(2000, (1 << 28) // (nx * ny)))
    steps = _log_int(rng, max(10, most_steps // 8), most_steps)
    return _resident(None, kind, nx, ny, storage, omega, steps, rng.random() < 0.3, rng.random() < 0.3)


# ---- inputs -------------------------------------------------------------------
def _plate(ny):
    return max(6, int(round(ny * 40 / 180)) // 2 * 2)


def _boundary(kind, nx, ny):
    if kind == "couette":
        return BU.couette_flow_boundary_conditions(nx, ny, U_WALL, 1.0)
    if kind == "poiseuille":
        return BU.poiseuille_flow_boundary_conditions(nx, ny, (1.0 + DELTA_RHO) / 3.0, 1.0 / 3.0)
    if kind == "channel":
        return BU.von_karman_boundary_conditions(nx, ny, 1.0, U_IN, _plate(ny), walls=True, plate_offset=1)
    if kind == "cavity":
        return BU.cavity_boundary_conditions(nx, ny, U_LID, 1.0)
    return None


def _equilibrium(rho, ux, uy):
    """f_eq[9, nx, ny] in plain float64 operations."""
    usq = 1.5 * (ux * ux + uy * uy)
    out = torch.empty((9,) + tuple(rho.shape), dtype=torch.float64, device=rho.device)
    for i in range(9):
        cu = CX[i] * ux + CY[i] * uy
        out[i] = W[i] * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - usq)
    return out


def _fields(kind, nx, ny, seed, device):
    """Start of a run: a long density wave of random phase, the flow's own velocity
    plus the seeded noise of the channel study, populations at equilibrium."""
    host = random.Random(seed)
    px, py = host.uniform(0, 2 * math.pi), host.uniform(0, 2 * math.pi)
    gen = torch.Generator(device=device)
    gen.manual_seed(int(seed) & 0x7FFFFFFF)
    x = torch.arange(nx, dtype=torch.float64, device=device)[:, None]
    y = torch.arange(ny, dtype=torch.float64, device=device)[None, :]
    amp = 0.01 if kind == "periodic" else 1e-3
    rho = 1.0 + amp * torch.sin(2 * math.pi * x / nx + px) * torch.cos(2 * math.pi * y / ny + py)
    u = torch.empty((nx, ny, 2), dtype=torch.float64, device=device)
    u.uniform_(-1e-3, 1e-3, generator=gen)
    if kind == "channel":
        u[..., 0] += U_IN
    f = _equilibrium(rho, u[..., 0], u[..., 1]).permute(1, 2, 0).contiguous()
    return f, rho.contiguous(), u


def _members(case):
    """(nx, ny, omega) of the channels of a batch, from the case alone."""
    rng = random.Random(case["layout"])
    out = []
    for _ in range(case["members"]):
        nx = rng.randint(case["nx_lo"], case["nx_hi"])
        ny = max(20, int(round(nx * rng.uniform(case["aspect_lo"], case["aspect_hi"]) / 2) * 2))
        out.append((nx, ny, rng.uniform(0.9, 1.6)))
    return out


def _probe(nx, ny):
    return (3 * nx // 4, ny // 2)


def prepare(case, seed):
    if case["path"] == "batch":
        members = []
        for j, (nx, ny, omega) in enumerate(_members(case)):
            f, rho, u = _fields("channel", nx, ny, seed * 1000 + j, "cuda")
            members.append(Member(nx, ny, omega, _boundary("channel", nx, ny), steps=case["steps"],
                                  probe=_probe(nx, ny) if case["probe"] else None, f0=f, rho0=rho, u0=u, seed=j))
        return {"case": case, "batch": Batch(members, storage=case["storage"])}
    nx, ny = case["nx"], case["ny"]
    boundary = _boundary(case["kind"], nx, ny)
    fields = _fields(case["kind"], nx, ny, seed, "cuda")
    if case["path"] == "resident":
        lat = Lattice(nx, ny, case["omega"], boundary, storage=case["storage"],
                      probe=_probe(nx, ny) if case["probe"] else None, probe_cap=case["steps"])
        return {"case": case, "lattice": lat, "fields": fields}
    if case["path"] == "host_step":
        fields = tuple(t.cpu().numpy() for t in fields)
    return {"case": case, "boundary": boundary, "fields": fields}


# ---- one pass -----------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["path"] == "resident":
        lat = state["lattice"]
        lat.set_state(*state["fields"])
        if case["graph"]:
            lat.step_graph(case["steps"])
        else:
            lat.step(case["steps"])
        out = list(lat.read())
        if case["probe"]:
            out.append(lat.probe_trace())
        return out
    if case["path"] == "batch":
        batch = state["batch"].start()
        if case["graph"]:
            batch.run_graph()
        else:
            batch.run()
        out = [t for j in range(len(batch.members)) for t in batch.read(j)]
        if case["probe"]:
            out += [batch.probe_trace(j) for j in range(len(batch.members))]
        return out
    return list(LBM.lattice_boltzmann_step(*state["fields"], case["omega"], state["boundary"]))


def work(case):
    """The state in (f, rho, u) and out, once each, and the operations of one BGK
    update (moments 20, equilibrium and relaxation 100) per node and step."""
    if case["path"] == "batch":
        nodes = sum(nx * ny for nx, ny, _ in _members(case))
    else:
        nodes = case["nx"] * case["ny"]
    return {"bytes": 2 * 96 * nodes, "flops": 120 * nodes * case.get("steps", 1)}


# ---- the same in plain float64 --------------------------------------------------
def _bounce(post, pre, x, y, dirs, speed=0.0):
    """f_post[opp i] = f_pre[i] - 6 w_i c_i.(speed, 0) on the nodes [x, y] for i in dirs."""
    for i in dirs:
        post[OPP[i]][x, y] = pre[i][x, y] - 6.0 * W[i] * CX[i] * speed


def _plain_boundary(kind, nx, ny, post, pre, prev):
    every = slice(None)
    if kind == "couette":
        _bounce(post, pre, every, -1, (2, 5, 6))
        _bounce(post, pre, every, 0, (4, 7, 8), U_WALL)
    elif kind == "poiseuille":
        _bounce(post, pre, every, 0, (4, 7, 8))
        _bounce(post, pre, every, -1, (2, 5, 6))
    elif kind == "cavity":
        _bounce(post, pre, 0, every, (3, 7, 6))
        _bounce(post, pre, -1, every, (1, 5, 8))
        _bounce(post, pre, every, 0, (4, 7, 8))
        _bounce(post, pre, every, -1, (2, 5, 6), U_LID)
    elif kind == "channel":
        one = torch.ones((1, 1), dtype=torch.float64, device=post.device)
        post[:, 0, :] = _equilibrium(one, U_IN * one, 0.0 * one)[:, 0]
        for i in (3, 6, 7):
            post[i][-1] = prev[i][-2]
        plate, px = _plate(ny), nx // 4
        low, high = ny // 2 - plate // 2 + 1, ny // 2 + plate // 2
        _bounce(post, pre, px, slice(low + 1, high), (1, 5, 8))
        _bounce(post, pre, px, high, (1, 8))
        _bounce(post, pre, px, low, (1, 5))
        _bounce(post, pre, px + 1, slice(low + 1, high), (3, 7, 6))
        _bounce(post, pre, px + 1, high, (3, 7))
        _bounce(post, pre, px + 1, low, (3, 6))
        _bounce(post, pre, every, 0, (4, 7, 8))
        _bounce(post, pre, every, -1, (2, 5, 6))


def _plain_moments(f):
    rho = f.sum(0)
    return rho, (f[1] + f[5] + f[8] - f[3] - f[6] - f[7]) / rho, (f[2] + f[5] + f[6] - f[4] - f[7] - f[8]) / rho


def _plain(kind, nx, ny, omega, steps, seed, probe):
    """f, rho, u after ``steps`` steps and the probe's velocities before each step but the first."""
    f, rho, u = _fields(kind, nx, ny, seed, "cuda")
    f = f.permute(2, 0, 1).contiguous()
    ux, uy = u[..., 0].clone(), u[..., 1].clone()
    trace = []
    for s in range(steps):
        if probe is not None and s > 0:
            trace.append(torch.stack([ux[probe], uy[probe]]))
        pre = _equilibrium(rho, ux, uy)
        if kind == "poiseuille":
            non_equilibrium = (1.0 - omega) * (f - pre)
        pre = f + (pre - f) * omega
        if kind == "poiseuille":
            for dst, src, target, dirs in ((0, -2, 1.0 + DELTA_RHO, (1, 5, 8)), (-1, 1, 1.0, (3, 6, 7))):
                feq = _equilibrium(torch.full_like(ux[src], target), ux[src], uy[src])
                for i in dirs:
                    pre[i][dst] = feq[i] + non_equilibrium[i][src]
        post = torch.stack([torch.roll(pre[i], (CX[i], CY[i]), (0, 1)) for i in range(9)])
        _plain_boundary(kind, nx, ny, post, pre, f)
        f = post
        rho, ux, uy = _plain_moments(f)
    out = [f.permute(1, 2, 0).contiguous(), rho, torch.stack([ux, uy], -1)]
    return out, (torch.stack(trace) if trace else None)


def exact(case, seed):
    if case["path"] == "batch":
        out, traces = [], []
        for j, (nx, ny, omega) in enumerate(_members(case)):
            o, t = _plain("channel", nx, ny, omega, case["steps"], seed * 1000 + j,
                          _probe(nx, ny) if case["probe"] else None)
            out += o
            traces.append(t)
        return out + (traces if case["probe"] else [])
    nx, ny = case["nx"], case["ny"]
    steps = case.get("steps", 1)
    probe = _probe(nx, ny) if case.get("probe") else None
    out, trace = _plain(case["kind"], nx, ny, case["omega"], steps, seed, probe)
    if case["path"] == "host_step":
        out = [t.cpu().numpy() for t in out]
    return out + ([trace] if probe is not None else [])
