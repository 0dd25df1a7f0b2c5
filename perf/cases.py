"""Performance cases of the framework, each through its public entry points.

A case is one call (or one training pass) of a program that a user of the stencil DSL runs:
explicit 2-D and 3-D sweeps, the lid-driven cavity in FP64 and in mixed precision, batches of
uneven problems, and a rollout with its gradients.  ``listed()`` names twelve of them, ``draw``
gives others of the same ranges, odd extents included.

Time levels live on the GPU; a pass returns the levels that the call wrote as device tensors,
which is how a program reads results without a copy to the host.
"""
import dataclasses
import math
import os

import numpy as np
import torch
import torch.utils.checkpoint

import xgrid
from xgrid_gb300.adjoint import Rollout

CACHE = os.path.join(".xgrid_cache", "perf")
float2d = xgrid.grid[float, 2]
float3d = xgrid.grid[float, 3]


# ------------------------------------------------------------------ programs
# Each body is ordinary DSL code.  In FP32 programs every coefficient is an argument: a Python
# literal is a C double and would promote the update to FP64.
def heat2d(u: float2d, c: float) -> None:
    u[0, 0] = u[0, 0] + c * (u[1, 0] + u[-1, 0] + u[0, 1] + u[0, -1] - 4.0 * u[0, 0])
    with xgrid.boundary(1):
        u[0, 0] = 0.0


def transport2d(u: float2d, a0: float, axm: float, axp: float, aym: float, ayp: float) -> None:
    u[0, 0] = a0 * u[0, 0] + axm * u[0, -1] + axp * u[0, 1] + aym * u[-1, 0] + ayp * u[1, 0]


def diffuse3d(u: float3d, k: float3d, dt: float) -> None:
    u[0, 0, 0] = u[0, 0, 0] + dt * ((k[0, 0, 0] + k[1, 0, 0]) * (u[1, 0, 0] - u[0, 0, 0]) +
                                    (k[0, 0, 0] + k[-1, 0, 0]) * (u[-1, 0, 0] - u[0, 0, 0]) +
                                    (k[0, 0, 0] + k[0, 1, 0]) * (u[0, 1, 0] - u[0, 0, 0]) +
                                    (k[0, 0, 0] + k[0, -1, 0]) * (u[0, -1, 0] - u[0, 0, 0]) +
                                    (k[0, 0, 0] + k[0, 0, 1]) * (u[0, 0, 1] - u[0, 0, 0]) +
                                    (k[0, 0, 0] + k[0, 0, -1]) * (u[0, 0, -1] - u[0, 0, 0]))


def walls3d(u: float3d, a0: float, a1: float, cold: float, hot: float) -> None:
    u[0, 0, 0] = a0 * u[0, 0, 0] + a1 * (u[1, 0, 0] + u[-1, 0, 0] + u[0, 1, 0] + u[0, -1, 0] +
                                         u[0, 0, 1] + u[0, 0, -1])
    with xgrid.boundary(1):
        u[0, 0, 0] = cold
    with xgrid.boundary(2):
        u[0, 0, 0] = hot


@dataclasses.dataclass
class Config:
    rho: float
    nu: float
    dt: float
    dx: float
    dy: float


def cavity(b: float2d, p: float2d, u: float2d, v: float2d, cfg: Config) -> None:
    b[0, 0] = (cfg.rho * (1.0 / cfg.dt *
                          ((u[0, 1] - u[0, -1]) / (2.0 * cfg.dx) + (v[1, 0] - v[-1, 0]) / (2.0 * cfg.dy)) -
                          ((u[0, 1] - u[0, -1]) / (2.0 * cfg.dx)) ** 2.0 -
                          2.0 * ((u[1, 0] - u[-1, 0]) / (2.0 * cfg.dy) * (v[0, 1] - v[0, -1]) / (2.0 * cfg.dx)) -
                          ((v[1, 0] - v[-1, 0]) / (2.0 * cfg.dy)) ** 2.0))

    p[0, 0] = (((p[0, 1] + p[0, -1]) * cfg.dy ** 2.0 + (p[1, 0] + p[-1, 0]) * cfg.dx ** 2.0) /
               (2.0 * (cfg.dx ** 2.0 + cfg.dy ** 2.0)) -
               cfg.dx ** 2.0 * cfg.dy ** 2.0 / (2.0 * (cfg.dx ** 2.0 + cfg.dy ** 2.0)) * b[0, 0][0])
    with xgrid.boundary(1):
        p[0, 0] = p[0, -1][0]
    with xgrid.boundary(2):
        p[0, 0] = p[1, 0][0]
    with xgrid.boundary(3):
        p[0, 0] = p[0, 1][0]
    with xgrid.boundary(4):
        p[0, 0] = 0.0

    for _ in range(0, 50):
        p[0, 0] = (((p[0, 1][0] + p[0, -1][0]) * cfg.dy ** 2.0 + (p[1, 0][0] + p[-1, 0][0]) * cfg.dx ** 2.0) /
                   (2.0 * (cfg.dx ** 2.0 + cfg.dy ** 2.0)) -
                   cfg.dx ** 2.0 * cfg.dy ** 2.0 / (2.0 * (cfg.dx ** 2.0 + cfg.dy ** 2.0)) * b[0, 0][0])
        with xgrid.boundary(1):
            p[0, 0] = p[0, -1][0]
        with xgrid.boundary(2):
            p[0, 0] = p[1, 0][0]
        with xgrid.boundary(3):
            p[0, 0] = p[0, 1][0]
        with xgrid.boundary(4):
            p[0, 0] = 0.0

    u[0, 0] = (u[0, 0] -
               u[0, 0] * cfg.dt / cfg.dx * (u[0, 0] - u[0, -1]) -
               v[0, 0] * cfg.dt / cfg.dy * (u[0, 0] - u[-1, 0]) -
               cfg.dt / (2.0 * cfg.rho * cfg.dx) * (p[0, 1][0] - p[0, -1][0]) +
               cfg.nu * (cfg.dt / cfg.dx ** 2.0 * (u[0, 1] - 2.0 * u[0, 0] + u[0, -1]) +
                         cfg.dt / cfg.dy ** 2.0 * (u[1, 0] - 2.0 * u[0, 0] + u[-1, 0])))

    v[0, 0] = (v[0, 0] -
               u[0, 0] * cfg.dt / cfg.dx * (v[0, 0] - v[0, -1]) -
               v[0, 0] * cfg.dt / cfg.dy * (v[0, 0] - v[-1, 0]) -
               cfg.dt / (2.0 * cfg.rho * cfg.dy) * (p[1, 0][0] - p[-1, 0][0]) +
               cfg.nu * (cfg.dt / cfg.dx ** 2.0 * (v[0, 1] - 2.0 * v[0, 0] + v[0, -1]) +
                         cfg.dt / cfg.dy ** 2.0 * (v[1, 0] - 2.0 * v[0, 0] + v[-1, 0])))

    with xgrid.boundary(1):
        u[0, 0] = 0.0
        v[0, 0] = 0.0
    with xgrid.boundary(2):
        u[0, 0] = 1.0


# --------------------------------------------------------------------- cases
def listed():
    return [
        # one step of a small explicit program: what a call costs (the 512 x 512 diffusion configuration)
        {"name": "heat2d_512", "kind": "heat2d", "ny": 512, "nx": 512},
        # the lid-driven cavity, one time step with its 51 pressure sweeps: a coarse run,
        # the headline size, and a size whose spacing is no power of two (divisions stay divisions)
        {"name": "cavity_257", "kind": "cavity", "n": 257, "mixed": False},
        {"name": "cavity_1025", "kind": "cavity", "n": 1025, "mixed": False},
        {"name": "cavity_1500", "kind": "cavity", "n": 1500, "mixed": False},
        # the fine cavity with FP32 defect correction of the pressure loop
        {"name": "cavity_mixed_4097", "kind": "cavity", "n": 4097, "mixed": True},
        # one step of a large FP32 field that streams from memory
        {"name": "transport2d_4096", "kind": "transport2d", "ny": 4096, "nx": 4096},
        # time loops over many uneven periodic problems: a sweep of parameters, and a handful
        {"name": "batch_60", "kind": "batch", "count": 60, "lo": 64, "hi": 1024, "steps": 96, "shapes": 1},
        {"name": "batch_8", "kind": "batch", "count": 8, "lo": 64, "hi": 512, "steps": 50, "shapes": 2},
        # variable-coefficient 3-D diffusion, one step: the benchmark cube, and ragged extents with clamped edges
        {"name": "diffuse3d_256", "kind": "diffuse3d", "nz": 256, "ny": 256, "nx": 256, "overstep": "wrap"},
        {"name": "diffuse3d_ragged", "kind": "diffuse3d", "nz": 203, "ny": 245, "nx": 307, "overstep": "limit"},
        # 3-D heat conduction in a box with cold walls and one hot wall (boundary masks)
        {"name": "walls3d_256", "kind": "walls3d", "nz": 256, "ny": 256, "nx": 256},
        # training pass: 20 diffusion steps, mean-square loss, gradients of the field and the coefficient
        {"name": "rollout_256", "kind": "rollout", "nz": 256, "ny": 256, "nx": 256, "steps": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["heat2d", "cavity", "mixed", "transport2d", "batch", "diffuse3d", "walls3d", "rollout"])
    if kind == "heat2d":
        return {"kind": kind, "ny": _log(rng, 64, 2048), "nx": _log(rng, 64, 2048)}
    if kind == "cavity":
        return {"kind": kind, "n": _log(rng, 65, 1500), "mixed": False}
    if kind == "mixed":
        return {"kind": "cavity", "n": _log(rng, 513, 4097), "mixed": True}
    if kind == "transport2d":
        return {"kind": kind, "ny": _log(rng, 256, 4096), "nx": _log(rng, 256, 4096)}
    if kind == "batch":
        hi = rng.randint(128, 1024)
        return {"kind": kind, "count": _log(rng, 4, 60), "lo": 64, "hi": hi, "steps": _log(rng, 8, 96),
                "shapes": rng.randint(3, 1 << 20)}
    nz, ny, nx = (_log(rng, 32, 256) for _ in range(3))
    if kind == "rollout":
        return {"kind": kind, "nz": nz, "ny": ny, "nx": nx, "steps": rng.randint(4, 20)}
    if kind == "diffuse3d":
        return {"kind": kind, "nz": nz, "ny": ny, "nx": nx, "overstep": rng.choice(["wrap", "limit"])}
    return {"kind": kind, "nz": nz, "ny": ny, "nx": nx}


def _shapes(case):
    rng = np.random.default_rng(case["shapes"])
    return [tuple(int(n) for n in rng.integers(case["lo"], case["hi"] + 1, 2)) for _ in range(case["count"])]


# -------------------------------------------------------------------- inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f32(x):
    return float(np.float32(x))


def _smooth(shape, gen, amplitude):
    """A smooth random FP64 field: a few sine modes of random wave number, phase and size."""
    y = torch.linspace(0.0, 1.0, shape[0], dtype=torch.float64, device=_device())[:, None]
    x = torch.linspace(0.0, 1.0, shape[1], dtype=torch.float64, device=_device())[None, :]
    f = torch.zeros(shape, dtype=torch.float64, device=_device())
    c = torch.rand((4, 5), dtype=torch.float64, generator=gen, device=_device()).tolist()
    for ky, kx, py, px, a in c:
        f += (a - 0.5) * torch.sin((1 + 3 * ky) * math.pi * y + 6 * py) * torch.sin((1 + 3 * kx) * math.pi * x + 6 * px)
    return f * amplitude


def _inputs(case, seed):
    """The fields (tensors) and scalar arguments of a case: the call's inputs, from the seed alone."""
    gen = torch.Generator(device=_device()).manual_seed(seed)
    host = np.random.default_rng(seed)

    def uniform(shape, dtype):
        return torch.rand(shape, dtype=dtype, generator=gen, device=_device())

    kind = case["kind"]
    if kind == "heat2d":
        return [uniform((case["ny"], case["nx"]), torch.float64)], (float(host.uniform(0.1, 0.24)),)
    if kind == "cavity":
        n = case["n"]
        h = 2.0 / (n - 1)
        nu = float(host.uniform(0.08, 0.12))
        # the time step at 0.13 h^2 / nu: 5e-6 at 1025 points, inside the explicit limits
        fields = [_smooth((n, n), gen, a) for a in (1.0, 0.1, 0.3, 0.3)]  # b, p, u, v
        fields[2][0] = fields[2][:, 0] = fields[2][:, -1] = 0.0
        fields[2][-1] = 1.0
        fields[3][0] = fields[3][-1] = fields[3][:, 0] = fields[3][:, -1] = 0.0
        return fields, (1.0, nu, 0.13 * h * h / nu, h, h)
    if kind in ("transport2d", "batch"):
        fields, values = [], []
        for shape in ([(case["ny"], case["nx"])] if kind == "transport2d" else _shapes(case)):
            cy, cx = host.uniform(-1.0, 1.0, 2)
            nu = host.uniform(0.01, 0.1)
            dy, dx = 1.0 / shape[0], 1.0 / shape[1]
            dt = 0.2 * min(dy, dx) ** 2 / nu
            gy, gx, ky, kx = 0.5 * cy * dt / dy, 0.5 * cx * dt / dx, nu * dt / (dy * dy), nu * dt / (dx * dx)
            fields.append(uniform(shape, torch.float32))
            values.append(tuple(_f32(a) for a in (1.0 - 2.0 * kx - 2.0 * ky, gx + kx, kx - gx, gy + ky, ky - gy)))
        return fields, values
    shape = (case["nz"], case["ny"], case["nx"])
    u = uniform(shape, torch.float32)
    if kind == "walls3d":
        a1 = _f32(host.uniform(0.1, 0.16))
        return [u], (_f32(1.0 - 6.0 * a1), a1, 0.0, 1.0)
    k = torch.exp(math.log(0.01) + math.log(10.0) * uniform(shape, torch.float32))
    fields = [u, k] + ([uniform(shape, torch.float32)] if kind == "rollout" else [])
    return fields, (_f32(0.8 / (12.0 * 0.1)),)


def _masks(case):
    kind = case["kind"]
    if kind == "heat2d":
        m = np.ones((case["ny"], case["nx"]), dtype=np.int32)
        m[1:-1, 1:-1] = 0
        return [m]
    if kind == "walls3d":
        m = np.ones((case["nz"], case["ny"], case["nx"]), dtype=np.int32)
        m[1:-1, 1:-1, 1:-1] = 0
        m[0] = 2
        return [m]
    if kind == "cavity":
        n = case["n"]
        wall = np.ones((n, n), dtype=np.int32)
        wall[1:-1, 1:-1] = 0
        u, p = wall.copy(), np.zeros((n, n), dtype=np.int32)
        u[-1, :] = 2
        p[:, -1] = 1
        p[0, :] = 2
        p[:, 0] = 3
        p[-1, :] = 4
        return [wall, p, u, wall]
    return None


# --------------------------------------------------------- kernels of a program
_kernels: dict = {}


def _kernel(case):
    """The compiled kernel (or rollout) of a program: made once, as a program does, and called for every state."""
    kind = case["kind"]
    options = {"precision": "float", "overstep": "none"}
    if kind in ("heat2d", "cavity"):
        options["precision"] = "double"
    if kind == "cavity" and case["mixed"]:
        options["mixed"] = "fp32"
    if kind in ("transport2d", "batch", "rollout"):
        options["overstep"] = "wrap"
    if kind == "diffuse3d":
        options["overstep"] = case["overstep"]
    xgrid.init(cacheroot=CACHE, opt_level=3, **options)
    key = (kind, case.get("steps") if kind == "rollout" else None) + tuple(sorted(options.items()))
    if key not in _kernels:
        body = {"heat2d": heat2d, "cavity": cavity, "transport2d": transport2d, "batch": transport2d,
                "diffuse3d": diffuse3d, "walls3d": walls3d, "rollout": diffuse3d}[kind]
        k = xgrid.kernel()(body)
        _kernels[key] = Rollout(k, case["steps"]) if kind == "rollout" else k
    return _kernels[key]


def prepare(case, seed):
    kernel = _kernel(case)
    fields, values = _inputs(case, seed)
    kind = case["kind"]
    if kind == "rollout":
        u0, k, target = fields
        return {"kind": kind, "kernel": kernel, "u0": u0.requires_grad_(True), "k": k.requires_grad_(True),
                "target": target, "values": values}
    masks = _masks(case)
    grids = []
    for i, f in enumerate(fields):
        g = xgrid.Grid(tuple(f.shape), float)
        if masks is not None:
            g.boundary = masks[i]
        grids.append(g)
    levels = [g.tensor(0) for g in grids]
    torch.cuda.synchronize()  # the grids' own stream has zeroed them
    for t, f in zip(levels, fields):
        t.copy_(f)
    torch.cuda.synchronize()
    if kind == "batch":
        return {"kind": kind, "kernel": kernel, "problems": [(g, *v) for g, v in zip(grids, values)],
                "grids": grids, "steps": case["steps"]}
    if kind == "cavity":
        return {"kind": kind, "kernel": kernel, "args": (*grids, Config(*values)), "outputs": grids}
    if kind == "transport2d":
        values = values[0]
    return {"kind": kind, "kernel": kernel, "args": (*grids, *values), "outputs": grids[:1]}


def run(state):
    if state["kind"] == "rollout":
        u = state["kernel"](state["u0"], {"k": state["k"]}, state["values"])
        loss = ((u - state["target"]) ** 2).mean()
        gu, gk = torch.autograd.grad(loss, [state["u0"], state["k"]])
        return {"u": u, "loss": loss, "grad_u": gu, "grad_k": gk}
    if state["kind"] == "batch":
        state["kernel"].batch(state["problems"], state["steps"])
        return [g.tensor(0) for g in state["grids"]]
    state["kernel"](*state["args"])
    return [g.tensor(0) for g in state["outputs"]]


# ---------------------------------------------------------------------- work
def work(case):
    """Bytes: each input field read once and each output field written once.  Flops: the additions,
    multiplications and divisions of the program's expressions, launch constants taken out."""
    kind = case["kind"]
    if kind == "heat2d":
        cells = case["ny"] * case["nx"]
        return {"bytes": 16.0 * cells, "flops": 7.0 * cells}
    if kind == "cavity":
        cells = case["n"] ** 2
        # p, u, v in; b, p, u, v out; source 19, pressure sweep 8 x 51, momentum 2 x 22
        return {"bytes": 56.0 * cells, "flops": (19.0 + 8.0 * 51 + 44.0) * cells}
    if kind == "transport2d":
        cells = case["ny"] * case["nx"]
        return {"bytes": 8.0 * cells, "flops": 9.0 * cells}
    if kind == "batch":
        cells = sum(ny * nx for ny, nx in _shapes(case))
        return {"bytes": 8.0 * cells, "flops": 9.0 * cells * case["steps"]}
    cells = case["nz"] * case["ny"] * case["nx"]
    if kind == "diffuse3d":
        return {"bytes": 12.0 * cells, "flops": 25.0 * cells}
    if kind == "walls3d":
        return {"bytes": 8.0 * cells, "flops": 8.0 * cells}
    # the field, the coefficient and the target in; the field and two gradients out; a forward
    # step (25) and its reverse (about twice that) per step
    return {"bytes": 24.0 * cells, "flops": 75.0 * cells * case["steps"]}


# --------------------------------------------------------------------- exact
def _shift(a, axis, s, overstep):
    """The neighbour at offset s along an axis: periodic or clamped."""
    if overstep == "wrap":
        return torch.roll(a, -s, axis)
    n = a.shape[axis]
    return a.index_select(axis, (torch.arange(n, device=a.device) + s).clamp_(0, n - 1))


def _diffuse(u, k, dt, overstep):
    acc = 0.0
    for axis in range(3):
        for s in (1, -1):
            acc = acc + (k + _shift(k, axis, s, overstep)) * (_shift(u, axis, s, overstep) - u)
    return u + dt * acc


def exact(case, seed):
    fields, values = _inputs(case, seed)
    fields = [f.double() for f in fields]
    kind = case["kind"]
    if kind == "heat2d":
        u, (c,) = fields[0], values
        out = torch.zeros_like(u)
        m = u[1:-1, 1:-1]
        out[1:-1, 1:-1] = m + c * (u[2:, 1:-1] + u[:-2, 1:-1] + u[1:-1, 2:] + u[1:-1, :-2] - 4.0 * m)
        return [out]
    if kind == "walls3d":
        u, (a0, a1, cold, hot) = fields[0], values
        out = torch.full_like(u, cold)
        i = slice(1, -1)
        out[i, i, i] = a0 * u[i, i, i] + a1 * (u[2:, i, i] + u[:-2, i, i] + u[i, 2:, i] + u[i, :-2, i] +
                                               u[i, i, 2:] + u[i, i, :-2])
        out[0] = hot
        return [out]
    if kind == "diffuse3d":
        return [_diffuse(fields[0], fields[1], values[0], case["overstep"])]
    if kind in ("transport2d", "batch"):
        outs = []
        for u, (a0, axm, axp, aym, ayp) in zip(fields, values):
            for _ in range(case.get("steps", 1)):
                u = (a0 * u + axm * torch.roll(u, 1, 1) + axp * torch.roll(u, -1, 1) +
                     aym * torch.roll(u, 1, 0) + ayp * torch.roll(u, -1, 0))
            outs.append(u)
        return outs
    if kind == "rollout":
        u0, k, target = (f.requires_grad_(True) for f in fields)
        if u0.numel() * case["steps"] > 1 << 26:
            chunk = torch.utils.checkpoint.checkpoint  # a step's temporaries are made again in reverse
        else:
            def chunk(f, *a, **_):
                return f(*a)
        u = u0
        for _ in range(case["steps"]):
            u = chunk(_diffuse, u, k, values[0], "wrap", use_reentrant=False)
        loss = ((u - target) ** 2).mean()
        gu, gk = torch.autograd.grad(loss, [u0, k])
        return {"u": u.detach(), "loss": loss.detach(), "grad_u": gu, "grad_k": gk}
    _, p, u, v = fields
    rho, nu, dt, dx, dy = values
    i = slice(1, -1)
    c, e, w, n, s = (i, i), (i, slice(2, None)), (i, slice(None, -2)), (slice(2, None), i), (slice(None, -2), i)
    b = torch.zeros_like(p)
    ux, uy, vx, vy = ((u[e] - u[w]) / (2 * dx), (u[n] - u[s]) / (2 * dy),
                      (v[e] - v[w]) / (2 * dx), (v[n] - v[s]) / (2 * dy))
    b[c] = rho * ((ux + vy) / dt - ux ** 2 - 2 * uy * vx - vy ** 2)
    den = 2 * (dx ** 2 + dy ** 2)
    for _ in range(51):
        q = torch.empty_like(p)
        q[c] = ((p[e] + p[w]) * dy ** 2 + (p[n] + p[s]) * dx ** 2) / den - dx ** 2 * dy ** 2 / den * b[c]
        q[1:-1, -1] = q[1:-1, -2]
        q[0, 1:] = q[1, 1:]
        q[:-1, 0] = q[:-1, 1]
        q[-1, :] = 0.0
        p = q
    out = []
    for f, g in ((u, (p[e] - p[w]) / dx), (v, (p[n] - p[s]) / dy)):
        r = torch.zeros_like(f)
        r[c] = (f[c] - u[c] * dt / dx * (f[c] - f[w]) - v[c] * dt / dy * (f[c] - f[s]) - dt / (2 * rho) * g +
                nu * dt * ((f[e] - 2 * f[c] + f[w]) / dx ** 2 + (f[n] - 2 * f[c] + f[s]) / dy ** 2))
        out.append(r)
    out[0][-1] = 1.0
    return [b, p, *out]
