"""The work that a user of the library has it do, as cases that can be timed and checked.

Every case is one rollout, derivative or training step through the package's public entry points:

- ``static``   a run of ``steps`` static steps (time_step + step) from an initial state; with ``limiter`` "learned" the
               slopes go through the network;
- ``moving``   a run on the moving mesh with the remesh on the device, from a mesh and a state;
- ``rollout``  the differentiable rollout: forward, then the backward to the initial state's gradient (checkpoints);
- ``jacobian`` one step's adjoint and tangent products from the same state (a solver's or a test's pair of products);
- ``lines``    a batch of 1D Riemann problems stepped together (the limiter's data factory), host state in and out;
- ``train``    one training step of the limiter's network: the gradient of a batch, then Adam.

Meshes are jittered lattices of unit-cubic cells (``mesh.jittered_points``), built on the device. States: ``blast`` (the
point blast: two cell widths of hot gas in a cold uniform box), ``acoustic`` (a plane sound wave of amplitude 1e-6),
``wave`` (waves in every primitive plus 1 % noise: no region is uniform), ``shear`` (the two-layer shear flow).

``exact`` evaluates the same map in plain torch float64: the mesh arrays are its input.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from luna_cpp_b200 import autograd, hydro
from luna_cpp_b200.learned import LimiterMLP, init_params, trained_params
from luna_cpp_b200.line import Line
from luna_cpp_b200.mesh import jittered_points
from luna_cpp_b200.remesh import Remesher

GAMMA = 5.0 / 3.0
COURANT = 0.3
LINE_GAMMA = 1.4
LINE_COURANT = 0.8
GRID = 2.0 ** -30  # the moving step's snapping grid, in box lengths
FACES_PER_CELL = {2: 3.0, 3: 7.95}  # of a jittered lattice
TRAIN_LR = 2e-3


def _static(name, cells, problem, precision="fp64", riemann="hllc", steps=4, limiter="plain"):
    nx, ny, nz = (list(cells) + [0])[:3]
    return {"name": name, "kind": "static", "nx": nx, "ny": ny, "nz": nz, "problem": problem, "precision": precision,
            "riemann": riemann, "steps": steps, "limiter": limiter}


def listed():
    return [
        # a latency-bound run: the mesh of a test or of one member of a parameter scan
        _static("static_blast_16", (16, 16, 16), "blast"),
        # the benchmark's step
        _static("static_blast_128", (128, 128, 128), "blast"),
        # an ordinary box of odd sides, HLL, limited everywhere
        _static("static_wave_odd", (61, 47, 53), "wave", riemann="hll"),
        # the reduced-precision benchmark: float face arithmetic and flux rows on a smooth wave
        _static("static_single_128", (128, 128, 128), "acoustic", precision="single"),
        # 2D runs in the reference's storage preset
        _static("static_shear_2d", (512, 384), "shear", precision="grad16"),
        # the learned limiter in a step, every cell through the network
        _static("static_learned_64", (64, 64, 64), "wave", limiter="learned"),
        # the moving-mesh benchmark: remesh, both flux passes
        {"name": "moving_blast_128", "kind": "moving", "nx": 128, "ny": 128, "nz": 128, "problem": "blast",
         "precision": "single", "steps": 2},
        # a 2D moving run in double
        {"name": "moving_wave_2d", "kind": "moving", "nx": 210, "ny": 150, "nz": 0, "problem": "wave", "precision": "fp64",
         "steps": 2},
        # a segment of the adjoint configuration's rollout (512^2, checkpointed)
        {"name": "rollout_2d", "kind": "rollout", "nx": 512, "ny": 512, "nz": 0, "problem": "wave", "steps": 8, "every": 4},
        # one step's products in 3D
        {"name": "jacobian_3d", "kind": "jacobian", "nx": 72, "ny": 64, "nz": 60, "problem": "wave", "riemann": "hllc"},
        # the limiter's 1D data: 1024-cell lines
        {"name": "lines_512", "kind": "lines", "cells": 1024, "lines": 512, "steps": 200, "walls": "outflow"},
        # one step of the limiter's training (the trainer's batch)
        {"name": "train_16k", "kind": "train", "rows": 16384},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, dim, lo, hi):
    """Sides of a box of about equal ones whose cell count is log-uniform."""
    base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return [max(lo, min(hi, int(round(base * rng.uniform(0.8, 1.2))))) for _ in range(dim)] + [0] * (3 - dim)


def draw(rng):
    kind = rng.choice(["static", "static", "static", "moving", "rollout", "jacobian", "lines", "train"])
    if kind == "static":
        dim = rng.choice([2, 3, 3])
        nx, ny, nz = _sides(rng, dim, 14, 120) if dim == 3 else _sides(rng, dim, 40, 900)
        precision = rng.choice(["fp64", "fp64", "fp32", "grad32", "grad16", "single"])
        problem = rng.choice(["blast", "acoustic", "wave"] if dim == 3 else ["blast", "wave", "shear"])
        learned = precision == "fp64" and problem == "wave" and rng.random() < 0.3
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "problem": problem, "precision": precision,
                "riemann": rng.choice(["hllc", "hll"]) if precision == "fp64" else "hllc", "steps": rng.randint(2, 5),
                "limiter": "learned" if learned else "plain"}
    if kind == "moving":
        dim = rng.choice([2, 3])
        nx, ny, nz = _sides(rng, dim, 16, 80) if dim == 3 else _sides(rng, dim, 48, 420)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "problem": rng.choice(["blast", "wave"]),
                "precision": rng.choice(["fp64", "fp32", "single"]), "steps": rng.randint(1, 3)}
    if kind == "rollout":
        dim = rng.choice([2, 2, 3])
        nx, ny, nz = _sides(rng, dim, 12, 40) if dim == 3 else _sides(rng, dim, 40, 500)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "problem": "wave", "steps": rng.randint(3, 8), "every": rng.randint(2, 5)}
    if kind == "jacobian":
        dim = rng.choice([2, 3, 3])
        nx, ny, nz = _sides(rng, dim, 12, 70) if dim == 3 else _sides(rng, dim, 40, 600)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "problem": "wave", "riemann": rng.choice(["hllc", "hll"])}
    if kind == "lines":
        cells = _log_int(rng, 100, 4000)
        return {"kind": kind, "cells": cells, "lines": _log_int(rng, 1, max(2, min(900, 1000000 // cells))),
                "steps": rng.randint(60, 200), "walls": rng.choice(["outflow", "reflective", "periodic"])}
    return {"kind": kind, "rows": _log_int(rng, 500, 250000)}


# ---- inputs -----------------------------------------------------------------------------------------------------------

def _box(case):
    n = [c for c in (case["nx"], case["ny"], case["nz"]) if c]
    return n, [c / n[0] for c in n]


def _points(case, seed):
    n, box = _box(case)
    pts = jittered_points(n, side=box, jitter=0.1, seed=1 + seed % (1 << 30))
    if case["kind"] == "moving":
        step = GRID * max(box)
        pts = np.round(pts / step) * step % np.asarray(box)
    return pts, box


def _conserved(W, volume, gamma=GAMMA):
    D = W.shape[-1] - 2
    rho, v, P = W[..., 0], W[..., 1:1 + D], W[..., D + 1]
    E = P / (gamma - 1) + 0.5 * rho * (v * v).sum(-1)
    return torch.cat([rho[..., None], rho[..., None] * v, E[..., None]], -1) * volume[..., None]


def _state(case, seed, cells, box):
    """Q [N, D + 2] on the device, from the cells' centroids and volumes and the seed."""
    dev = torch.device("cuda")
    rng = torch.Generator(device=dev)
    rng.manual_seed(7919 * (seed + 1))
    volume = torch.tensor(cells.volume, device=dev)
    c = torch.tensor(cells.positions + cells.centroid, device=dev)
    side = torch.tensor(box, dtype=torch.float64, device=dev)
    N, D = c.shape
    x = (c / side) % 1.0
    a = torch.rand(12, generator=rng, device=dev, dtype=torch.float64)
    k = 2 * math.pi
    W = torch.zeros(N, D + 2, dtype=torch.float64, device=dev)
    if case["problem"] == "blast":
        h = float(side.prod() / N) ** (1.0 / D)
        r = (((x - 0.5) * side) ** 2).sum(1).sqrt()
        inside = r < 2.0 * h
        W[:, 0] = 1.0
        W[:, D + 1] = 1e-5
        q = _conserved(W, volume)
        q[:, D + 1] += torch.where(inside, (0.5 + a[0]) * volume / volume[inside].sum(), torch.zeros_like(volume))
        return q
    if case["problem"] == "acoustic":
        s = 1e-6 * (0.5 + a[0]) * torch.sin(k * (x[:, 0] + a[1]))
        W[:, 0] = 1.0 + s
        W[:, 1] = s
        W[:, D + 1] = 0.6 + s
        return _conserved(W, volume)
    if case["problem"] == "shear":
        inner = (x[:, 1] - 0.5).abs() < 0.25
        W[:, 0] = torch.where(inner, 2.0, 1.0)
        W[:, 1] = torch.where(inner, 0.5, -0.5)
        modes = torch.arange(1, 9, dtype=torch.float64, device=dev)
        amp = torch.randn(8, generator=rng, device=dev, dtype=torch.float64)
        W[:, 2] = 0.01 * (amp * torch.sin(k * modes * x[:, :1])).sum(1)
        W[:, D + 1] = 2.5
        return _conserved(W, volume)
    noise = 0.02 * (torch.rand(N, D + 2, generator=rng, device=dev, dtype=torch.float64) - 0.5)
    W[:, 0] = 1 + 0.2 * torch.sin(k * (x[:, 0] + a[0]))
    W[:, 1] = 0.3 * torch.sin(k * (x[:, 1] + a[1]))
    W[:, 2] = 0.2 * torch.cos(k * (x[:, D - 1] + a[2]))
    if D == 3:
        W[:, 3] = 0.25 * torch.sin(k * (x[:, 0] + x[:, 2] + a[3]))
    W[:, D + 1] = 1 + 0.2 * torch.cos(k * (x.sum(1) + a[4]))
    return _conserved(W + noise, volume)


def _line_inputs(case, seed):
    """Riemann problems of the training distribution on one jittered line: positions [n], Q [lines, n, 3]."""
    rng = np.random.default_rng(seed)
    n, B = case["cells"], case["lines"]
    x = (np.arange(n) + 0.5 + rng.uniform(-0.1, 0.1, n)) / n
    gap, _ = _line_gaps(x, case["walls"] == "periodic")
    volume = 0.5 * (gap[:-1] + gap[1:])
    rho = np.exp(rng.uniform(np.log(0.1), np.log(10), (B, 2)))
    u = rng.uniform(-1, 1, (B, 2))
    p = np.exp(rng.uniform(np.log(0.01), np.log(10), (B, 2)))
    right = (x > rng.uniform(0.4, 0.6, (B, 1))).astype(np.int64)
    pick = np.arange(B)[:, None], right
    r, v, P = rho[pick], u[pick], p[pick]
    q = np.stack([r, r * v, P / (LINE_GAMMA - 1) + 0.5 * r * v * v], -1) * volume[None, :, None]
    return x, np.ascontiguousarray(q)


def _line_gaps(x, periodic):
    """The distances between the line's points (and over its ends) on the solver's 2^-52 grid."""
    key = np.rint(x * 2.0 ** 52)
    inner = np.diff(key)
    ends = (key[0] + 2.0 ** 52 - key[-1],) * 2 if periodic else (2 * key[0], 2 * (2.0 ** 52 - key[-1]))
    return np.concatenate([[ends[0]], inner, [ends[1]]]) * 2.0 ** -52, key * 2.0 ** -52


def _line_walls(case):
    periodic = case["walls"] == "periodic"
    wall = "outflow" if periodic else case["walls"]
    return {"walls": (wall, wall), "periodic": periodic}


def _train_inputs(case, seed):
    rng = torch.Generator(device="cuda")
    rng.manual_seed(104729 * (seed + 1))
    n = case["rows"]
    x = (2 * torch.rand(n, 32, generator=rng, device="cuda") - 1).to(torch.bfloat16)
    f = x[:, :5].float()
    t = (0.5 + 0.4 * torch.tanh(f - 0.5 * x[:, 5:10].float())).contiguous()
    w = (torch.rand(n, 5, generator=rng, device="cuda") > 0.2).float()
    return x, t, w, init_params(seed % 1000)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, t, w, p = _train_inputs(case, seed)
        return {"case": case, "x": x, "t": t, "w": w, "net": LimiterMLP(p)}
    if kind == "lines":
        x, q = _line_inputs(case, seed)
        return {"case": case, "q": q, "line": Line(x, 1.0, lines=case["lines"], gamma=LINE_GAMMA, **_line_walls(case))}
    pts, box = _points(case, seed)
    start = Remesher(len(box), box)
    mesh = start.build(pts)
    q0 = _state(case, seed, mesh.cells(), box)
    s = {"case": case, "q0": q0, "start": start, "mesh": mesh}
    if kind == "moving":
        s["fv"] = hydro.FiniteVolume(mesh, precision=case["precision"], motion="moving")
        s["remesher"] = Remesher(len(box), box)
        return s
    s["fv"] = hydro.FiniteVolume(mesh, precision=case.get("precision", "fp64"), riemann=case.get("riemann", "hllc"))
    if case.get("limiter") == "learned":
        s["fv"].set_limiter("learned", torch.tensor(trained_params(), device="cuda"))
    if kind == "jacobian":
        s["qbar"], s["dq"] = _directions(seed, q0)
    return s


def _directions(seed, q0):
    rng = torch.Generator(device="cuda")
    rng.manual_seed(15485863 * (seed + 1))
    qbar, d = (torch.randn(q0.shape, generator=rng, device="cuda", dtype=torch.float64) for _ in range(2))
    return qbar, d * q0[:, :1]


class _DeviceArray:
    """Device memory of the library as torch sees it."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": "<f8", "version": 3}


def _copy(ptr, shape):
    """A tensor of the caller's own: the library's memory is only the mesh's until the next build."""
    return torch.as_tensor(_DeviceArray(ptr, shape), device="cuda").clone()


# ---- one pass ---------------------------------------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        net = s["net"]
        loss = net.gradient(s["x"], s["t"], s["w"])
        net.adam(lr=TRAIN_LR)
        return {"loss": loss, "grad": net.grad, "params": net.params}
    if kind == "lines":
        ln = s["line"]
        ln.set_state(s["q"])
        dt = ln.time_step(LINE_COURANT, "luna")
        for _ in range(case["steps"]):
            dt = ln.step_and_time_step(dt, LINE_COURANT)
        return {"q": ln.get_state(), "dt": dt}
    fv, q0 = s["fv"], s["q0"]
    if kind == "rollout":
        q = q0.detach().requires_grad_(True)
        out = autograd.rollout(q, fv, case["steps"], COURANT, case["every"])
        autograd.kinetic_y(out).backward()
        return {"q": out.detach(), "grad": q.grad, "dt": autograd.last_dts(out)}
    if kind == "jacobian":
        fv.set_state(q0)
        dt = fv.time_step(COURANT)
        qbar = fv.step_adjoint(dt, s["qbar"].clone())
        dq = fv.step_tangent(dt, s["dq"].clone())
        return {"qbar": qbar, "dq": dq, "q": fv.get_state(torch.empty_like(q0)), "dt": dt}
    dts = []
    if kind == "moving":
        fv.set_mesh(s["mesh"])
        fv.set_state(q0)
        for _ in range(case["steps"]):
            dt = fv.time_step(COURANT)
            dts.append(dt)
            mesh = fv.step_moving_device(dt, s["remesher"])
        N, D = mesh.n_cells, mesh.dim
        return {"q": fv.get_state(torch.empty_like(q0)), "dt": dts, "positions": _copy(mesh.desc.positions, (N, D)),
                "volume": _copy(mesh.desc.volume, (N,)), "centroid": _copy(mesh.desc.centroid, (N, D))}
    fv.set_state(q0)
    for _ in range(case["steps"]):
        dt = fv.time_step(COURANT)
        dts.append(dt)
        fv.step(dt)
    return {"q": fv.get_state(torch.empty_like(q0)), "dt": dts}


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

def _step_work(case):
    """One static step: the whole-mesh dt comes between the sweep and the update, so the mesh and the state are read once
    before it and once after it, and the gradients go through memory."""
    D = 3 if case["nz"] else 2
    N = case["nx"] * case["ny"] * max(1, case["nz"])
    V, fpc = D + 2, FACES_PER_CELL[D]
    grad = {"fp64": 8, "grad16": 2}.get(case.get("precision", "fp64"), 4) * V * D
    face = 8 + 16 * D  # cells, area, centroid
    sweep = 8 * V + 8 + 16 * D + 4 + 8 * fpc + face * fpc + grad
    fluxes = face * fpc + 8 * V + grad + 16 * D + 8 + 8 * V
    flops = fpc * (488 if D == 3 else 300) + 2 * fpc * V * (4 * D + 6)
    return N, (sweep + fluxes) * N, flops * N


def work(case):
    kind = case["kind"]
    if kind == "train":
        n, p = case["rows"], 32 * 64 + 64 * 64 + 64 * 16
        return {"bytes": n * (64 + 40) + 28 * (p + 144), "flops": 6 * n * p}
    if kind == "lines":
        n = case["cells"] * case["lines"]
        return {"bytes": n * 48 * case["steps"] + 48 * n, "flops": n * 250 * case["steps"]}
    N, step_bytes, step_flops = _step_work(case)
    D = 3 if case["nz"] else 2
    V, fpc = D + 2, FACES_PER_CELL[D]
    state = 16 * V * N  # the state set and read back
    if kind == "moving":
        mesh = N * (fpc * (8 + 16 * D + 8) + 4 + 24 * D)  # the new mesh written once
        second = N * (fpc * (8 + 16 * D) + 16 * V + 24 * D)
        return {"bytes": case["steps"] * (step_bytes + mesh + second) + state, "flops": case["steps"] * N * fpc * (1000 if D == 3 else 500)}
    if kind == "rollout":  # forward, forward again, adjoint (the step's inputs and bars, both ways)
        return {"bytes": case["steps"] * 4 * step_bytes + state, "flops": case["steps"] * 5 * step_flops}
    if kind == "jacobian":  # the adjoint, the tangent, the step
        return {"bytes": 5 * step_bytes + state, "flops": 6 * step_flops}
    learned = (N * (64 + 40 + 40) * 2, N * 14000) if case["limiter"] == "learned" else (0, 0)
    return {"bytes": case["steps"] * (step_bytes + learned[0]) + state, "flops": case["steps"] * (step_flops + learned[1])}


def tolerance(case):
    """About four times what the same path shows with its state perturbed at its own rounding (1e-15, or 3e-8 where the
    slopes or the Riemann solve are float), or against ``exact``, rounded up to a power of ten where the sizes vary."""
    kind, precision = case["kind"], case.get("precision", "fp64")
    if kind == "train":
        return {"rel": 4e-3}  # BF16 operands: the gradient is 1e-3 off exact's
    if kind in ("lines", "rollout", "jacobian"):
        return {"rel": 1e-13, "max": 1e-11}  # 1e-14 and, of the bars, 3e-13 seen
    if precision in ("fp32", "single") and case["problem"] == "blast":
        # a float Riemann solve across the blast's front (a pressure ratio of 1e9) cancels: one rounding of the state moves
        # the cells that the front has just reached by a part in a hundred (5e-4 and 0.65 seen)
        return {"rel": 2e-3, "max": 0.99}
    if kind == "moving":
        # a rounding can move a generator by one step of the 2^-30 grid, which is up to 1e-6 of a centroid's offset
        return {"rel": 1e-6, "max": 1e-5} if precision != "fp64" else {"rel": 1e-9, "max": 1e-5}
    if case["limiter"] == "learned":
        return {"rel": 4e-5}  # BF16 features and weights: 1e-5 off exact's
    if precision == "grad16":
        return {"rel": 1e-6, "max": 1e-4}  # a float slope at a binary16 rounding boundary
    if precision == "grad32":
        return {"rel": 1e-7, "max": 1e-5}
    if precision in ("fp32", "single"):
        return {"rel": 2e-7, "max": 1e-6}
    return {"rel": 1e-13, "max": 1e-11}


# ---- the same in plain torch float64 ----------------------------------------------------------------------------------

class _Exact:
    """One static MUSCL-Hancock step over mesh arrays (luna-cpp's src/hydro/finite_volume.hpp:463-641, :1277-1435,
    :1538-1631), vectorised over faces; differentiable."""

    def __init__(self, mesh, riemann, gamma=GAMMA, net=None):
        dev = torch.device("cuda")
        self.gamma, self.riemann, self.net = gamma, riemann, net

        def put(a):
            return torch.as_tensor(np.ascontiguousarray(a), device=dev)

        o, j = put(mesh.owner).long(), put(mesh.neighbour).long()
        self.N, self.D = mesh.n_cells, mesh.dim
        self.V = self.D + 2
        box = torch.tensor(mesh.box, dtype=torch.float64, device=dev)
        pos, cen, self.vol = put(mesh.positions), put(mesh.centroid), put(mesh.volume)
        area, fcen = put(mesh.area), put(mesh.face_centroid)

        def wrap(d):
            return d - box * torch.round(d / box)

        d = wrap(pos[j] - pos[o])
        self.o, self.j, self.d = o, j, d
        self.dist = d.square().sum(1).sqrt()
        self.mag = area.square().sum(1).sqrt()
        self.n = torch.where(self.mag[:, None] > 0, area / self.mag[:, None].clamp_min(1e-300), torch.zeros_like(area))
        self.off = [fcen - cen[o], fcen - d - cen[j]]
        self.radius = (self.vol * (3 / (4 * math.pi))) ** (1 / 3) if self.D == 3 else (self.vol / math.pi).sqrt()
        surface = torch.zeros_like(self.vol).index_add_(0, o, self.mag).index_add_(0, j, self.mag)
        self.keep = [self.mag >= 1e-6 * surface[c] for c in (o, j)]
        # the fit's operator rows: g_i = sum_k c_k (W_k - W_i)
        U = self.D + 1
        one = torch.ones_like(self.mag)[:, None]
        X = [torch.cat([one, d + cen[j] - cen[o]], 1), torch.cat([one, -d + cen[o] - cen[j]], 1)]
        M = torch.zeros(self.N, U * U, dtype=torch.float64, device=dev)
        for x, i in zip(X, (o, j)):
            M.index_add_(0, i, (self.mag[:, None, None] * x[:, :, None] * x[:, None, :]).reshape(-1, U * U))
        inv = torch.linalg.inv(M.reshape(-1, U, U))[:, 1:, :]
        self.c = [torch.einsum("fap,fp->fa", inv[i], self.mag[:, None] * x) for x, i in zip(X, (o, j))]

    def primitive(self, q):
        U = q / self.vol[:, None]
        rho = U[:, :1].clamp_min(1e-10)
        v = U[:, 1:-1] / rho
        floor = 1e-20 / self.gamma / (self.gamma - 1)
        e = torch.maximum(U[:, -1:] - 0.5 * rho * (v * v).sum(1, keepdim=True), floor * rho)
        return torch.cat([rho, v, (self.gamma - 1) * e], 1)

    def sides(self):
        return ((self.o, self.j), (self.j, self.o))

    def gradients(self, W):
        N, V, D = self.N, self.V, self.D
        g = W.new_zeros(N, V * D)
        big = torch.finfo(torch.float64).max
        lo, hi = W.new_full((N, V), big), W.new_full((N, V), -big)
        for s, (i, k) in enumerate(self.sides()):
            g = g.index_add(0, i, ((W[k] - W[i])[:, :, None] * self.c[s][:, None, :]).reshape(-1, V * D))
            keep = self.keep[s][:, None]
            lo = lo.scatter_reduce(0, i[:, None].expand(-1, V), torch.where(keep, W[k], W.new_full((), big)), "amin")
            hi = hi.scatter_reduce(0, i[:, None].expand(-1, V), torch.where(keep, W[k], W.new_full((), -big)), "amax")
        g = g.reshape(N, V, D)
        cap = 1.0 if self.net is None else 2.0
        phi = W.new_full((N, V), cap)
        for s, (i, k) in enumerate(self.sides()):
            dp = (g[i] * self.off[s][:, None, :]).sum(2)
            room = torch.where(dp > 0, hi[i] - W[i], W[i] - lo[i]).clamp_min(0.0)
            f = torch.where(dp != 0, room / torch.where(dp != 0, dp.abs(), torch.ones_like(dp)), W.new_full((), cap))
            f = torch.where(self.keep[s][:, None], f.clamp_max(cap), W.new_full((), cap))
            phi = phi.scatter_reduce(0, i[:, None].expand(-1, V), f, "amin")
        if self.net is not None:
            phi = phi * torch.sigmoid(self.logits(W, g, lo, hi, phi))
        return g * phi[:, :, None]

    def logits(self, W, g, lo, hi, alpha):
        """The limiter's network on its features (luna_cpp_b200/learned.py): density slot 0, velocities 1.., pressure 4."""
        D = self.D
        slot = [0] + list(range(1, D + 1)) + [4]
        rng = hi - lo
        scale = W.abs() + hi.abs() + lo.abs()
        safe = torch.maximum(rng, 1e-12 * scale)
        f = W.new_zeros(self.N, 32)
        c = (self.gamma * W[:, -1] / W[:, 0]).sqrt()
        for v, k in enumerate(slot):
            f[:, 4 * k] = alpha[:, v] / 2
            f[:, 4 * k + 1] = ((W[:, v] - lo[:, v]) / safe[:, v]).clamp(-1, 2) - 0.5
            f[:, 4 * k + 2] = torch.tanh(g[:, v].square().sum(1).sqrt() * self.radius / safe[:, v])
            f[:, 4 * k + 3] = torch.tanh(3 * rng[:, v] / scale[:, v])
        f[:, 20] = torch.tanh(torch.log(hi[:, -1] / lo[:, -1]))
        f[:, 21] = torch.tanh(W[:, 1:-1].square().sum(1).sqrt() / c)
        f[:, 22] = alpha.amin(1).clamp_max(1.0)
        f[:, 23] = 1.0
        return _mlp(self.net, f)[:, slot]

    def time_step(self, W):
        c = (self.gamma * W[:, -1] / W[:, 0]).sqrt()
        v = W[:, 1:-1]
        vsig = c[self.o] + c[self.j] - ((v[self.j] - v[self.o]) * self.d).sum(1) / self.dist
        r = torch.minimum(self.radius[self.o], self.radius[self.j])
        face = torch.where(vsig > 0, (self.dist + r) / vsig.clamp_min(1e-300), torch.full_like(vsig, 1e300)).min()
        cell = (self.radius / (c + v.square().sum(1).sqrt())).min()
        return float(COURANT * torch.minimum(face, cell))

    def face_state(self, W, g, rate, i, r, dt):
        Wf = W[i] - 0.5 * dt * rate[i] + (g[i] * r[:, None, :]).sum(2)
        ok = (Wf[:, 0] > 0) & (Wf[:, -1] > 0)
        return torch.where(ok[:, None], Wf, W[i])

    def rate(self, W, g):
        D = self.D
        rho, v, P = W[:, 0], W[:, 1:-1], W[:, -1]
        div = sum(g[:, 1 + a, a] for a in range(D))

        def along(k):
            return (v * g[:, k]).sum(1)

        rows = [along(0) + rho * div] + [along(1 + a) + g[:, D + 1, a] / rho for a in range(D)] + [along(D + 1) + self.gamma * P * div]
        return torch.stack(rows, 1)

    def flux(self, L, R, n):
        g1 = self.gamma

        def side(W):
            vn = (W[:, 1:-1] * n).sum(1)
            E = W[:, -1] / (g1 - 1) + 0.5 * W[:, 0] * W[:, 1:-1].square().sum(1)
            m = W[:, 0] * vn
            F = torch.cat([m[:, None], m[:, None] * W[:, 1:-1] + W[:, -1:] * n, ((E + W[:, -1]) * vn)[:, None]], 1)
            U = torch.cat([W[:, :1], W[:, :1] * W[:, 1:-1], E[:, None]], 1)
            return vn, (g1 * W[:, -1] / W[:, 0]).sqrt(), E, F, U

        vl, cl, El, Fl, Ul = side(L)
        vr, cr, Er, Fr, Ur = side(R)
        SL, SR = torch.minimum(vl - cl, vr - cr), torch.maximum(vl + cl, vr + cr)
        if self.riemann == "hll":
            mid = (SR[:, None] * Fl - SL[:, None] * Fr + (SL * SR)[:, None] * (Ur - Ul)) / (SR - SL)[:, None]
            return torch.where((SL >= 0)[:, None], Fl, torch.where((SR <= 0)[:, None], Fr, mid))
        dl, dr = L[:, 0] * (SL - vl), R[:, 0] * (SR - vr)
        SM = (R[:, -1] - L[:, -1] + dl * vl - dr * vr) / (dl - dr)

        def star(W, S, vn, E, den, F, U):
            rho = den / (S - SM)
            e = E / W[:, 0] + (SM - vn) * (SM + W[:, -1] / den)
            Us = torch.cat([rho[:, None], rho[:, None] * (W[:, 1:-1] + n * (SM - vn)[:, None]), (rho * e)[:, None]], 1)
            return F + S[:, None] * (Us - U)

        left = torch.where((SL >= 0)[:, None], Fl, star(L, SL, vl, El, dl, Fl, Ul))
        right = torch.where((SR <= 0)[:, None], Fr, star(R, SR, vr, Er, dr, Fr, Ur))
        return torch.where(((SL >= 0) | (SM >= 0))[:, None], left, right)

    def step(self, q, dt=None):
        W = self.primitive(q)
        if dt is None:
            dt = self.time_step(W.detach())
        g = self.gradients(W)
        rate = self.rate(W, g)
        L = self.face_state(W, g, rate, self.o, self.off[0], dt)
        R = self.face_state(W, g, rate, self.j, self.off[1], dt)
        F = self.flux(L, R, self.n) * self.mag[:, None]
        return q.index_add(0, self.o, -dt * F).index_add(0, self.j, dt * F), dt


def _mlp(p, x):
    """The 32-64-64-16 network with the flat parameters p, float64."""
    w1, b1, w2, b2, w3, b3 = torch.split(p, [2048, 64, 4096, 64, 1024, 16])
    h = torch.relu(x @ w1.reshape(64, 32).T + b1)
    h = torch.relu(h @ w2.reshape(64, 64).T + b2)
    return h @ w3.reshape(16, 64).T + b3


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "lines":
        return _exact_lines(case, seed)
    if kind == "moving":
        return None  # a periodic Voronoi mesh of each step's generators in numpy takes minutes
    pts, box = _points(case, seed)
    remesher = Remesher(len(box), box)
    mesh = remesher.build(pts).to_host()
    q = _state(case, seed, mesh, box)
    net = torch.tensor(trained_params(), device="cuda", dtype=torch.float64) if case.get("limiter") == "learned" else None
    E = _Exact(mesh, case.get("riemann", "hllc"), net=net)
    if kind == "jacobian":
        qbar, dq = _directions(seed, q)
        x = q.clone().requires_grad_(True)
        out, dt = E.step(x)
        u = qbar.clone().requires_grad_(True)
        (vjp,) = torch.autograd.grad(out, x, u, create_graph=True)
        (jvp,) = torch.autograd.grad(vjp, u, dq)
        return {"qbar": vjp.detach(), "dq": jvp.detach(), "q": out.detach(), "dt": dt}
    dts = []
    if kind == "rollout":
        x = q.clone().requires_grad_(True)
        out = x
        for _ in range(case["steps"]):
            out, dt = E.step(out)
            dts.append(dt)
        (grad,) = torch.autograd.grad((out[:, 2] ** 2 / out[:, 0]).sum(), x)
        return {"q": out.detach(), "grad": grad, "dt": dts}
    with torch.no_grad():
        for _ in range(case["steps"]):
            q, dt = E.step(q)
            dts.append(dt)
    return {"q": q, "dt": dts}


def _exact_train(case, seed):
    x, t, w, p = _train_inputs(case, seed)
    p = torch.tensor(p, device="cuda", dtype=torch.float64, requires_grad=True)
    w = w.double()
    o = _mlp(p, x.double())[:, :5]
    loss = (w * (torch.sigmoid(o) - t.double()) ** 2).sum() / w.sum()
    (g,) = torch.autograd.grad(loss, p)
    # the first Adam step from zero moments: m / (1 - beta1) = g, v / (1 - beta2) = g^2
    return {"loss": loss.detach().reshape(1), "grad": g, "params": p.detach() - TRAIN_LR * g / (g.abs() + 1e-8)}


def _exact_lines(case, seed):
    """The 1D step (luna-cpp's src/hydro/finite_volume_1d.hpp:117-206, :332-384, :492-660) over all lines at once."""
    x, q = _line_inputs(case, seed)
    dev, gamma = torch.device("cuda"), LINE_GAMMA
    periodic, wall = case["walls"] == "periodic", case["walls"]
    gap, _ = _line_gaps(x, periodic)
    gap = torch.tensor(gap, device=dev)
    volume = 0.5 * (gap[:-1] + gap[1:])
    cen = 0.25 * (gap[1:] - gap[:-1])
    q = torch.tensor(q, device=dev)
    n = volume.numel()

    def pad(a, mirror):
        """[.., n, k] with one cell beyond each end: the other end's, or the end cell itself (velocity mirrored)."""
        if periodic:
            return torch.cat([a[:, -1:], a, a[:, :1]], 1)
        m = torch.tensor([1.0, -1.0, 1.0], device=dev, dtype=torch.float64) if mirror else 1.0
        return torch.cat([a[:, :1] * m, a, a[:, -1:] * m], 1)

    c = torch.cat([cen[-1:], cen, cen[:1]]) if periodic else torch.cat([-cen[:1], cen, -cen[-1:]])

    def primitive(q):
        U = q / volume[:, None]
        rho = U[..., 0].clamp_min(1e-10)
        v = U[..., 1] / rho
        e = torch.maximum(U[..., 2] - 0.5 * rho * v * v, rho * (1e-20 / gamma / (gamma - 1)))
        return torch.stack([rho, v, (gamma - 1) * e], -1)

    def time_step(q):
        W = primitive(q)
        a = (gamma * W[..., 2] / W[..., 0]).sqrt()
        return (LINE_COURANT * volume / (W[..., 1].abs() + a)).amin(1)

    dL = (-gap[:-1] + c[:-2] - cen)[:, None]
    dR = (gap[1:] + c[2:] - cen)[:, None]
    rL, rR = (-0.5 * gap[:-1] - cen)[:, None], (0.5 * gap[1:] - cen)[:, None]

    def clip(g, r, room_hi, room_lo):
        dp = g * r
        safe = torch.where(dp != 0, dp, torch.ones_like(dp))
        up = (dp > 0) & (dp > room_hi)
        down = (dp < 0) & (dp < room_lo)
        return torch.where(up, g * (room_hi.clamp_min(0.0) / safe), torch.where(down, g * (room_lo.clamp_max(0.0) / safe), g))

    def flux(L, R):
        vl, vr = L[..., 1], R[..., 1]
        cl, cr = (gamma * L[..., 2] / L[..., 0]).sqrt(), (gamma * R[..., 2] / R[..., 0]).sqrt()
        SL, SR = torch.minimum(vl - cl, vr - cr), torch.maximum(vl + cl, vr + cr)
        dl, dr = L[..., 0] * (SL - vl), R[..., 0] * (SR - vr)
        SM = (R[..., 2] - L[..., 2] + dl * vl - dr * vr) / (dl - dr)

        def side(W, S, den, outer):
            v, E = W[..., 1], W[..., 2] / (gamma - 1) + 0.5 * W[..., 0] * W[..., 1] ** 2
            F = torch.stack([W[..., 0] * v, W[..., 0] * v * v + W[..., 2], (E + W[..., 2]) * v], -1)
            U = torch.stack([W[..., 0], W[..., 0] * v, E], -1)
            rho = den / (S - SM)
            e = E / W[..., 0] + (SM - v) * (SM + W[..., 2] / den)
            star = F + S[..., None] * (torch.stack([rho, rho * SM, rho * e], -1) - U)
            return torch.where(outer[..., None], F, star)

        left = side(L, SL, dl, SL >= 0)
        right = side(R, SR, dr, SR <= 0)
        return torch.where(((SL >= 0) | (SM >= 0))[..., None], left, right)

    def step(q, dt):
        W = primitive(q)
        P = pad(W, wall == "reflective")
        left, right = P[:, :-2] - W, P[:, 2:] - W
        g = (right - left) / (dR - dL)
        hi, lo = torch.maximum(left, right), torch.minimum(left, right)
        g = clip(g, rL, hi, lo)
        g = clip(g, rR, hi, lo)
        rho, v, p = W.unbind(-1)
        rate = torch.stack([v * g[..., 0] + rho * g[..., 1], v * g[..., 1] + g[..., 2] / rho, gamma * p * g[..., 1] + v * g[..., 2]], -1)
        half = W - 0.5 * dt[:, None, None] * rate

        def face(r):
            f = half + g * r
            return torch.where(((f[..., 0] > 0) & (f[..., 2] > 0))[..., None], f, W)

        fl, fr = face(rL), face(rR)  # each cell's states at its two faces
        m = torch.tensor([1.0, -1.0, 1.0], device=dev, dtype=torch.float64)
        if periodic:
            first, last = fr[:, -1:], fl[:, :1]
        elif wall == "reflective":
            first, last = fl[:, :1] * m, fr[:, -1:] * m
        else:
            first, last = W[:, :1], W[:, -1:]
        F = flux(torch.cat([first, fr], 1), torch.cat([fl, last], 1))
        return q - dt[:, None, None] * (F[:, 1:] - F[:, :-1])

    dt = time_step(q)
    for _ in range(case["steps"]):
        q = step(q, dt)
        dt = time_step(q)
    return {"q": q.cpu().numpy(), "dt": dt.cpu().numpy()}
