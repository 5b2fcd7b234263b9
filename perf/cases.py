"""What a user of this solver has it do, as cases to be timed.

A case is one of four kinds, each through the package's public classes:

  run      CLbmSolverGB300.run: `steps` time steps of one cavity, then density
           and velocity to the host, as the `lbm_gb300` program does between two
           visualisation outputs (the configurations write one every 100 steps)
  stepped  the same with alternating simulationStepAlpha / simulationStepBeta
           calls, the reference's own time loop (the drop-in use)
  batch    LbmBatch.run over cavities of the seeded batch workload, then every
           cavity's fields to the host
  serve    an LbmServer that gets a set of requests, runs its rounds until all
           are done and hands out their results

Lid speed, viscosity and the starting flow come from the seed.  A later pass on
the same state continues the simulation (run, stepped, batch) or submits the
same requests again (serve).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from cavityflow_cuda_gb300.solver import CLbmSolverGB300, LbmBatch, LbmServer
from cavityflow_cuda_gb300.workloads import SERVE_EDGES, SERVE_WEIGHTS, MT19937_64, batch_workload, lattice_tau

# D3Q19 in the solver's order: 0 +x, 1 -x, 2 +y, 3 -y, 4 +x+y, 5 -x-y, 6 +x-y, 7 -x+y, 8 +x+z, 9 -x-z, 10 +x-z,
# 11 -x+z, 12 +y+z, 13 -y-z, 14 +y-z, 15 -y+z, 16 +z, 17 -z, 18 rest.
C = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (1, 1, 0), (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1),
     (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1), (0, 0, 1), (0, 0, -1),
     (0, 0, 0)]
W = [1 / 3 if k == 18 else 1 / 18 if k < 4 or k >= 16 else 1 / 36 for k in range(19)]
OPP = [18 if k == 18 else k ^ 1 for k in range(19)]
PERIOD = 16  # planes after which the starting flow repeats along z


def _single(kind, size, storage, steps, lid="injection", fma=False):
    return {"kind": kind, "nx": size[0], "ny": size[1], "nz": size[2], "storage": storage,
            "steps": steps, "lid": lid, "fma": fma}


def listed():
    return [
        # the 64^3 FP64 configuration (Re = 100), the one the golden results are held to
        {"name": "cavity64_f64"} | _single("run", (64, 64, 64), "f64", 100),
        # the smallest cube of the serving workload, alone: launches and latency count
        {"name": "cavity32_f32"} | _single("run", (32, 32, 32), "f32", 200),
        # the 64^3 configuration in the default precision
        {"name": "cavity64_f32"} | _single("run", (64, 64, 64), "f32", 200),
        # the drop-in time loop on a box with no round edge, mass-conserving lid
        {"name": "stepped101_f32"} | _single("stepped", (101, 67, 83), "f32", 100, lid="wall"),
        # an ordinary cube in the 16-bit mode that meets the accuracy target
        {"name": "cavity128_f16sr"} | _single("run", (128, 128, 128), "f16sr", 100),
        # odd sizes and an odd number of steps, so that runs start on either kind of step
        {"name": "cavity193_f32"} | _single("run", (193, 200, 187), "f32", 101),
        # the other 16-bit storage
        {"name": "cavity256_bf16s"} | _single("run", (256, 256, 256), "bf16s", 100),
        # the 384^3 benchmark configuration
        {"name": "cavity384_f32"} | _single("run", (384, 384, 384), "f32", 100),
        # the 512^3 precision workload
        {"name": "cavity512_f16sr"} | _single("run", (512, 512, 512), "f16sr", 100),
        # part of the 512-cavity batch workload, in FP32
        {"name": "batch64_f32", "kind": "batch", "count": 64, "storage": "f32", "steps": 100, "workload": 0},
        # the whole batch workload in 16 bits
        {"name": "batch512_f16sr", "kind": "batch", "count": 512, "storage": "f16sr", "steps": 200, "workload": 0},
        # requests of the serving workload's sizes with short step counts
        {"name": "serve24_f16sr", "kind": "serve", "count": 24, "storage": "f16sr", "steps": 200, "workload": 1},
    ]


def draw(rng):
    storage = rng.choices(["f32", "f16sr", "f64", "f16s", "bf16s"], [6, 4, 3, 2, 2])[0]
    kind = rng.choices(["run", "stepped", "batch", "serve"], [11, 3, 3, 2])[0]
    if kind == "batch":
        count = round(math.exp(rng.uniform(math.log(4), math.log(64 if storage == "f64" else 512))))
        return {"kind": kind, "count": count, "storage": storage, "workload": rng.randrange(1 << 20),
                "steps": rng.randint(20, 30 if storage == "f64" else 200)}
    if kind == "serve":
        return {"kind": kind, "count": rng.randint(2, 28), "storage": storage, "workload": rng.randrange(1 << 20),
                "steps": rng.randint(20, 40 if storage == "f64" else 300)}
    most = {"f64": 160, "f32": 360}.get(storage, 480)
    while True:  # an edge of the cube of the same volume, spread over the logarithm; each axis up to 2 times off
        edge = math.exp(rng.uniform(math.log(16), math.log(most)))
        size = [max(8, round(edge * math.exp(rng.uniform(-math.log(2), math.log(2))))) for _ in range(3)]
        if size[0] * size[1] * size[2] <= most ** 3:
            break
    return _single(kind, size, storage, rng.randint(20, 30 if storage == "f64" else 100),
                   lid=rng.choices(["injection", "wall"], [4, 1])[0],
                   fma=storage in ("f32", "f64") and rng.random() < 0.25)


# -- inputs -----------------------------------------------------------------

def _flow(seed):
    """Lid speed and viscosity in lattice units: around the benchmark's 0.05 and 0.0192 .. 0.064."""
    r = random.Random(seed)
    return 0.03 + 0.04 * r.random(), 0.0192 * (0.064 / 0.0192) ** r.random()


def _start(case, seed, device):
    """PERIOD planes of starting populations (19, PERIOD, ny, nx) in the host value type: the equilibrium of a smooth
    seeded flow plus a small disturbance."""
    nx, ny = case["nx"], case["ny"]
    r = random.Random(seed + 1)
    ph = [2 * math.pi * r.random() for _ in range(6)]
    two_pi = 2 * math.pi
    x = torch.arange(nx, device=device, dtype=torch.float64)[None, None, :] * (two_pi / nx)
    y = torch.arange(ny, device=device, dtype=torch.float64)[None, :, None] * (two_pi / ny)
    z = torch.arange(PERIOD, device=device, dtype=torch.float64)[:, None, None] * (two_pi / PERIOD)
    u = [0.02 * torch.sin(x + ph[0]) * torch.cos(2 * y + ph[1]) + 0.0 * z,
         0.02 * torch.cos(2 * x + ph[2]) * torch.sin(y + ph[3]) * torch.cos(z),
         0.01 * torch.sin(x + y + z + ph[4]) + 0.0 * x]
    rho = 1 + 0.003 * torch.cos(x + ph[5]) * torch.cos(y) + 0.0 * z
    u2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    f = torch.empty((19, PERIOD, ny, nx), device=device,
                    dtype=torch.float64 if case["storage"] == "f64" else torch.float32)
    for k, c in enumerate(C):
        cu = c[0] * u[0] + c[1] * u[1] + c[2] * u[2]
        noise = torch.rand(rho.shape, generator=gen, device=device, dtype=torch.float32).double() - 0.5
        f[k] = W[k] * (rho + 3 * cu + 4.5 * cu * cu - 1.5 * u2 + 1e-3 * noise)
    return f


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=torch.float64 if dtype == np.float64 else torch.float32, pin_memory=True).numpy()


def _domains(case, seed):
    """(size, inv_tau, lid) of cavities of the batch workload; lid and viscosity are the seed's."""
    T = np.float64 if case["storage"] == "f64" else np.float32
    out = []
    for i, c in enumerate(batch_workload(count=case["count"], seed=case["workload"])):
        lid, nu = _flow(seed * 1009 + i)
        out.append((c.size, lattice_tau(nu, case["storage"])[1], float(T(lid))))
    return out


def _requests(case, seed):
    """(size, inv_tau, lid, steps) of requests with the serving workload's edges (up to 128) and weights."""
    r = MT19937_64(case["workload"])
    T = np.float64 if case["storage"] == "f64" else np.float32
    out = []
    for i in range(case["count"]):
        edge = min(128, SERVE_EDGES[r.choice(SERVE_WEIGHTS)])
        steps = r.integer(max(1, case["steps"] // 4), case["steps"])
        lid, nu = _flow(seed * 1009 + i)
        out.append(((edge, edge, edge), lattice_tau(nu, case["storage"])[1], float(T(lid)), steps))
    return out


def _groups(sizes, dtype):
    """Pinned space for the fields of cavities of these sizes, as at most 16 arrays, and each cavity's part of it."""
    n = -(-len(sizes) // 16)
    groups, parts = [], []
    for i in range(0, len(sizes), n):
        cells = [4 * s[0] * s[1] * s[2] for s in sizes[i:i + n]]
        groups.append(_pinned((sum(cells),), dtype))
        at = np.cumsum([0] + cells)
        parts += [groups[-1][at[k]:at[k + 1]].reshape(4, s[2], s[1], s[0]) for k, s in enumerate(sizes[i:i + n])]
    return groups, parts


def prepare(case, seed):
    dtype = np.float64 if case["storage"] == "f64" else np.float32
    if case["kind"] == "batch":
        doms = _domains(case, seed)
        batch = LbmBatch(doms, storage=case["storage"])
        groups, parts = _groups([d[0] for d in doms], dtype)
        return {"case": case, "batch": batch, "views": [batch.domain(i) for i in range(len(doms))],
                "groups": groups, "parts": parts}
    if case["kind"] == "serve":
        return {"case": case, "requests": _requests(case, seed),
                "server": LbmServer(budget_bytes=4 << 30, storage=case["storage"])}
    lid, nu = _flow(seed)
    n = (case["nx"], case["ny"], case["nz"])
    s = CLbmSolverGB300(n, lattice_tau(nu, case["storage"])[1], float(dtype(lid)), storage=case["storage"],
                        fused_multiply_add=case["fma"], lid=case["lid"])
    f = _start(case, seed, "cuda").cpu().numpy()
    for z in range(0, n[2], PERIOD):
        planes = min(PERIOD, n[2] - z)
        part = f if planes == PERIOD else np.ascontiguousarray(f[:, :planes])
        s.setDensityDistributions(part, (1, 1, 1 + z), (n[0], n[1], planes))
    state = {"case": case, "solver": s, "rho": _pinned((n[2], n[1], n[0]), dtype),
             "u": _pinned((3, n[2], n[1], n[0]), dtype)}
    if n[0] * n[1] * n[2] <= 64 ** 3:  # a small cavity's populations go to the host too (a checkpoint's content)
        state["f"] = _pinned((19, n[2], n[1], n[0]), dtype)
    return state


# -- one pass ---------------------------------------------------------------

def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].run(case["steps"])
        for v, f in zip(state["views"], state["parts"]):
            v.getDensities(out=f[0])
            v.getVelocities(out=f[1:])
        return state["groups"]
    if case["kind"] == "serve":
        srv = state["server"]
        ids = [srv.submit(*r) for r in state["requests"]]
        left, got = len(ids), {}
        while left:
            srv.round()
            for c in srv.poll():
                got[c["id"]] = srv.take_result(c["id"])
                left -= 1
        return [got[i] for i in ids]
    s = state["solver"]
    if case["kind"] == "stepped":
        for i in range(case["steps"] // 2):
            s.simulationStepAlpha()
            s.simulationStepBeta()
    else:
        s.run(case["steps"])
    out = {"rho": s.getDensities(out=state["rho"]), "u": s.getVelocities(out=state["u"])}
    if "f" in state:
        out["f"] = s.getDensityDistributions(out=state["f"])
    return out


def _cells(case):
    """(cells, steps) of each cavity of the case."""
    if case["kind"] == "batch":
        return [(s[0] * s[1] * s[2], case["steps"]) for s, _, _ in _domains(case, 0)]
    if case["kind"] == "serve":
        return [(s[0] * s[1] * s[2], n) for s, _, _, n in _requests(case, 0)]
    return [(case["nx"] * case["ny"] * case["nz"], case["steps"])]


def work(case):
    """The populations read once and written once, density and velocity written once; about 200 operations a cell and
    step (the moments, nine equilibrium pairs, the relaxation)."""
    s = {"f64": 8, "f32": 4}.get(case["storage"], 2)
    v = 8 if case["storage"] == "f64" else 4
    cells = _cells(case)
    n = sum(c for c, _ in cells)
    held = 1 if case["kind"] == "serve" else 2  # a served request starts at rest: nothing to read
    return {"bytes": n * (held * 19 * s + 4 * v), "flops": sum(200 * c * t for c, t in cells)}


# -- the same in 64 bits, in torch ------------------------------------------

def _cavity64(size, inv_tau, lid_u, steps, start=None, lid="injection"):
    """Density, velocity and the populations that arrive next, after `steps` D3Q19 steps (f <- f + (feq - f) / tau,
    then streaming) of a box with full-way bounce-back walls one cell outside the cavity and a lid that is either a row
    y = ny held at feq(1, (U, 0, 0)) or a moving wall above it."""
    nx, ny, nz = size
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    shape = (nz + 2, ny + 2, nx + 2)
    inner = (slice(1, -1),) * 3
    f = [torch.full(shape, W[k], dtype=torch.float64, device=dev) for k in range(19)]  # what arrives at each cell
    if start is not None:
        for k in range(19):
            for z in range(0, nz, PERIOD):
                n = min(PERIOD, nz - z)
                f[k][1 + z:1 + z + n, 1:-1, 1:-1] = start[k, :n].to(dev, torch.float64)
    post = f
    for _ in range(steps):
        if lid == "wall":
            f[5][1:-1, -2, 1:-1] -= lid_u / 6
            f[6][1:-1, -2, 1:-1] += lid_u / 6
        a = [t[inner] for t in f]
        rho = a[18].clone()
        j = [torch.zeros_like(rho) for _ in range(3)]
        for k in range(18):
            rho += a[k]
            for d in range(3):
                if C[k][d]:
                    j[d].add_(a[k], alpha=C[k][d])
        p = rho - 1.5 * (j[0] * j[0] + j[1] * j[1] + j[2] * j[2])
        post = []
        for k in range(19):
            e = p
            if k < 18:
                cu = sum(C[k][d] * j[d] for d in range(3) if C[k][d])
                e = p + cu * (3 + 4.5 * cu)
            t = f[OPP[k]].clone()  # a wall cell sends back what it got
            t[inner] = a[k] + inv_tau * (W[k] * e - a[k])
            if lid == "injection":
                cu = C[k][0] * lid_u
                t[1:-1, -2, 1:-1] = W[k] * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * lid_u * lid_u)
            post.append(t)
        f = [torch.roll(post[k], (C[k][2], C[k][1], C[k][0]), (0, 1, 2)) for k in range(19)]
    rho = sum(t[inner] for t in post)
    u = torch.stack([sum(C[k][d] * post[k][inner] for k in range(19) if C[k][d]) for d in range(3)])
    if lid == "injection":
        rho[:, -1, :] = 1
        u[:, :, -1, :] = 0
        u[0, :, -1, :] = lid_u
    return rho, u, torch.stack([t[inner] for t in f]) if nx * ny * nz <= 64 ** 3 else None


def exact(case, seed):
    if case["kind"] == "batch":
        if case["count"] > 64:
            return None
        got = [_cavity64(s, it, u, case["steps"]) for s, it, u in _domains(case, seed)]
        groups, parts = _groups([d[0] for d in _domains(case, seed)], np.float64)
        for part, (rho, u, _) in zip(parts, got):
            part[0], part[1:] = rho.cpu().numpy(), u.cpu().numpy()
        return groups
    if case["kind"] == "serve":
        return [tuple(x.cpu().numpy() for x in _cavity64(s, it, u, n)[:2]) for s, it, u, n in _requests(case, seed)]
    dtype = np.float64 if case["storage"] == "f64" else np.float32
    lid, nu = _flow(seed)
    start = _start(case, seed, "cuda" if torch.cuda.is_available() else "cpu")
    steps = case["steps"] // 2 * 2 if case["kind"] == "stepped" else case["steps"]
    rho, u, f = _cavity64((case["nx"], case["ny"], case["nz"]), lattice_tau(nu, case["storage"])[1],
                          float(dtype(lid)), steps, start, case["lid"])
    out = {"rho": rho.cpu().numpy(), "u": u.cpu().numpy()}
    if f is not None:  # after an odd step the slots hold what left the cells, not what arrives
        out["f"] = f.cpu().numpy() if steps % 2 == 0 else None
    return out
