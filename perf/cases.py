"""Workloads for timing the framework through its public entry points.

Four families, each a thing that a program built on this package does over and over:

  cell   one indented cell (core.CellSim): an output interval of `steps` time steps, then what an
         output reads back — the node positions, the indenter force and, with `fields`, the von
         Mises stress and pressure of every tetrahedron (Simulation.run reads the same).
  batch  many cells of uneven size and material advanced together (core.Batch), then the indenter
         force of every cell: how the surrogate's force curves are made.
  mlp    the surrogate's network (mlp.MLP) called forward, or forward and backward with the
         parameter gradients read back.
  learn  its long calls: minibatch training ("train") and fitting its inputs to curves ("fit").

A case is a dict of plain values; `listed` gives the fixed ones, `draw` random ones of the same
ranges. `prepare` builds the inputs and the handle from a seed, `run` makes one pass, `work` counts
the bytes and operations that a pass cannot do without, `exact` computes a pass's results in 64
bits with plain torch.

Quantities that the device holds in single precision (stress fields) and force readouts are
returned in single precision, as the surrogate's training set keeps its curves; positions are
returned as the getters give them.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from nofluidx3d_gb300.core import (CONTACT_PLANE, CONTACT_SPHERE, CONTACT_SUBSTRATE, FIELD_PRESSURE, FIELD_VON_MISES,
                                   Batch, CellSim)
from nofluidx3d_gb300.mesh import kuhn_sphere, mesh_counts
from nofluidx3d_gb300.mlp import MLP
from nofluidx3d_gb300.workloads import Workload

SPHERE_INTEGRAL = 3  # NFX_CONTACT_SPHERE_INTEGRAL
SETTLE_STEPS = 200   # the indenter advances over the first steps and then holds
SPEED = 1e-3         # indenter descent per step
DEPTH0 = 0.005       # indentation at time 0
MATERIALS = ("nh", "mr", "svk", "svkk", "vp")


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def listed() -> list[dict]:
    def cell(name, radius, material, steps, indenter="sphere", integrator="vv", fields=False):
        return dict(name=name, kind="cell", radius=radius, material=material, indenter=indenter,
                    integrator=integrator, steps=steps, fields=fields)

    return [
        # a coupling loop that reads the cell after every single step: launches and latency
        cell("cell_r4_one_step", 4.0, "mr", 1),
        # the small Neo-Hookean cell under a flat indenter, one output interval (workloads.plain_small)
        cell("cell_r8_interval", 8.0, "nh", 100, indenter="plane"),
        # the less common options together at an odd size and an odd interval: Saint-Venant-Kirchhoff,
        # the integrated sphere contact, lumped masses
        cell("cell_r21_options", 21.3, "svk", 37, indenter="sphere_integral", integrator="vv2"),
        # the 1M-tetra viscoplastic cell, one frame with its stress fields (workloads.plain_large_1m)
        cell("cell_r34_frame", 34.0, "vp", 100, fields=True),
        # a large elastic cell under a flat indenter
        cell("cell_r48_elastic", 48.0, "mr", 50, indenter="plane"),
        # the 6.6M-tetra viscoplastic cell, one output interval (workloads.plain_large)
        cell("cell_r64_interval", 64.0, "vp", 100),
        # many small cells in one launch: a chunk of a surrogate data set
        dict(name="batch_512_small", kind="batch", cells=512, r_lo=4.0, r_hi=8.0, meshes=12, steps=100,
             points=False),
        # cells of very uneven size and material together, their positions read back as well
        dict(name="batch_24_uneven", kind="batch", cells=24, r_lo=6.0, r_hi=32.0, meshes=24, steps=50, points=True),
        # the surrogate asked for a handful of curves
        dict(name="mlp_forward_37", kind="mlp", op="forward", width=256, depth=3, n_out=64, rows=37, max_batch=1024),
        # a hand-written training step of a wider network on an odd batch: losses, input and
        # parameter gradients
        dict(name="mlp_backward_wide", kind="mlp", op="backward", width=512, depth=5, n_out=128, rows=1000,
             max_batch=1000),
        # training the surrogate (6 -> 256 x 3 -> 64, minibatches of 512)
        dict(name="train_256", kind="learn", op="train", width=256, depth=3, n_out=64, rows=6144, batch=512,
             steps=256),
        # proposing material inputs for a chunk of curves (surrogate.propose: 16 starts per target)
        dict(name="fit_1024", kind="learn", op="fit", width=256, depth=3, n_out=64, rows=1024, batch=1024,
             steps=400),
    ]


def draw(rng) -> dict:
    def logu(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(("cell", "cell", "cell", "batch", "mlp", "learn"))
    if kind == "cell":
        radius = round(logu(3.0, 56.0), 2)
        material = rng.choice(MATERIALS)
        steps = max(1, round(logu(1.0, 250.0 if radius < 40.0 else 60.0)))
        return dict(kind="cell", radius=radius, material=material,
                    indenter=rng.choice(("plane", "sphere", "sphere", "sphere_integral")),
                    integrator=rng.choice(("vv", "vv", "vv2")), steps=steps,
                    fields=material == "vp" and rng.random() < 0.5)
    if kind == "batch":
        lo = round(logu(3.0, 10.0), 2)
        cells = round(logu(2.0, 512.0))
        hi = round(min(lo * rng.uniform(1.0, 3.0), 8.0 if cells > 100 else 26.0), 2)
        return dict(kind="batch", cells=cells, r_lo=min(lo, hi), r_hi=max(lo, hi), meshes=min(cells, 12),
                    steps=max(1, round(logu(5.0, 120.0))),
                    points=cells <= 32)
    width, depth, n_out = 16 * round(logu(2.0, 40.0)), rng.randint(1, 6), 8 * round(logu(1.0, 24.0))
    if kind == "mlp":
        rows = round(logu(1.0, 4096.0))
        return dict(kind="mlp", op=rng.choice(("forward", "backward")), width=width, depth=depth, n_out=n_out,
                    rows=rows, max_batch=rows)
    batch = round(logu(16.0, 1024.0))
    op = rng.choice(("train", "fit"))
    return dict(kind="learn", op=op, width=min(width, 384), depth=min(depth, 4), n_out=n_out,
                rows=batch if op == "fit" else batch * rng.randint(1, 8) + rng.randint(0, 15), batch=batch,
                steps=round(logu(8.0, 200.0)))


# ------------------------------------------------------------------------------------------
# cells and batches: set-up shared by prepare and exact
# ------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _mesh(radius: float, jitter_seed: int = 0):
    return kuhn_sphere(radius, 0.02, jitter_seed)


def _cell_workload(case: dict) -> Workload:
    return Workload("cell", radius=case["radius"], material="mr_vp" if case["material"] == "vp" else "mr")


def _elastic(material: str) -> tuple[int, float, float, float]:
    """(model, E, nu, Mooney-Rivlin ratio) of an elastic material."""
    mu, K = 1.2e-3, 1e-2
    E, nu = 9.0 * K * mu / (3.0 * K + mu), (3.0 * K - 2.0 * mu) / (2.0 * (3.0 * K + mu))
    return {"nh": 0, "mr": 0, "svk": 1, "svkk": 2}[material], E, nu, 0.8 if material == "mr" else 1.0


def _contacts(x: np.ndarray, indenter: str, radius: float) -> list[dict]:
    """A substrate tangent to the lower pole (node 4) of the positions x and an indenter already
    DEPTH0 into the upper one (node 3), descending for SETTLE_STEPS steps and then holding (the
    schedules of the workloads)."""
    top, bottom = float(x[3, 1]), float(x[4, 1])
    out = [dict(kind=CONTACT_SUBSTRATE, k=0.1, radius=0.0, p0=bottom, v=0.0, tmove=float("inf"))]
    Rs = max(0.25 * radius, 1.5)
    if indenter == "plane":
        out.append(dict(kind=CONTACT_PLANE, k=0.1, radius=0.0, p0=top - DEPTH0, v=SPEED, tmove=float(SETTLE_STEPS)))
    elif indenter == "sphere":
        out.append(dict(kind=CONTACT_SPHERE, k=0.1, radius=Rs, p0=top + Rs - DEPTH0, v=SPEED,
                        tmove=float(SETTLE_STEPS)))
    else:  # its force density decays over 1/k beyond the sphere: start clear of the cell
        out.append(dict(kind=SPHERE_INTEGRAL, k=12.0, radius=Rs, p0=top + Rs + 0.5, v=SPEED,
                        tmove=float(SETTLE_STEPS)))
    return out


def _deformed(mesh, rng) -> np.ndarray:
    """Positions of a cell in mid-indentation: long waves of half a percent of strain."""
    x = mesh.points
    u = np.zeros_like(x)
    for _ in range(3):
        k = rng.normal(size=3)
        k *= math.pi / (max(mesh.radius, 1.0) * np.linalg.norm(k))
        a = rng.normal(size=3)
        a *= 3e-3 / (np.linalg.norm(a) * np.linalg.norm(k))
        u += np.sin(x @ k + rng.uniform(0, 2 * math.pi))[:, None] * a
    return x + u


def _cell_state(case: dict, seed: int):
    """(mesh, positions, velocities, plastic tensor or None, contacts) of a cell case."""
    rng = np.random.default_rng([seed, 1])
    mesh = _mesh(case["radius"])
    x = _deformed(mesh, rng)
    v = 1e-4 * (_deformed(mesh, rng) - mesh.points)
    fp = None
    if case["material"] == "vp" and case["radius"] < 40.0:  # larger cells start from Fp = I
        nt = mesh.num_tetra
        fp = (np.eye(3).reshape(9, 1) + rng.normal(0.0, 5e-4, (9, nt))).reshape(-1)
    return mesh, x, v, fp, _contacts(x, case["indenter"], case["radius"])


def _batch_cells(case: dict, seed: int):
    """Per cell: mesh, its index among the distinct meshes, viscoplastic parameters, contacts."""
    rng = np.random.default_rng([seed, 2])
    radii = np.exp(np.linspace(math.log(case["r_lo"]), math.log(case["r_hi"]), case["meshes"]))
    which = np.sort(np.concatenate([np.arange(case["meshes"]),
                                    rng.integers(0, case["meshes"], case["cells"] - case["meshes"])]))
    out = []
    for i in which:
        R = round(float(radii[i]), 3)
        mesh = _mesh(R, int(i) + 1)
        mu = math.exp(rng.uniform(math.log(2e-4), math.log(2e-3)))
        ratio = math.exp(rng.uniform(math.log(5.0), math.log(20.0)))
        Y = math.exp(rng.uniform(math.log(5e-5), math.log(1e-3)))
        eta = math.exp(rng.uniform(math.log(1e-2), math.log(1e-1)))
        par = (0.8 * mu, 0.2 * mu, mu * ratio, 1.0, Y, Y / eta, 1.0, 0.0)
        out.append((mesh, int(i), par, _contacts(mesh.points, "sphere", R)))
    return out


def _prepare_cell(case: dict, seed: int):
    mesh, x, v, fp, contacts = _cell_state(case, seed)
    s = CellSim(0)
    s.set_mesh(mesh.points, mesh.tets)
    if case["material"] == "vp":
        s.set_viscoplastic(_cell_workload(case).vp_params())
    else:
        s.set_tetra(*_elastic(case["material"]))
    for c in contacts:
        s.add_contact(c["kind"], c["k"], c["radius"], c["p0"], c["v"], c["tmove"])
    if case["integrator"] == "vv2":
        s.set_integrator_lumped(0.05, 1.0)
    else:
        s.set_integrator(0.01, False)
    s.set_record(1, max(case["steps"], 20), 16384)
    s.set_points(x)
    s.set_velocities(v)
    if fp is not None:
        s.set_plastic_tensor_soa(fp)
    return {"case": case, "sim": s, "points": np.empty(3 * s.np)}


def _run_cell(state):
    case, s = state["case"], state["sim"]
    s.step(case["steps"])
    out = {"force": np.float32(s.indenter_force(1)), "points": s.points_soa(state["points"])}
    if case["fields"]:
        out["von_mises"] = s.tet_field(FIELD_VON_MISES).astype(np.float32)
        out["pressure"] = s.tet_field(FIELD_PRESSURE).astype(np.float32)
    return out


def _prepare_batch(case: dict, seed: int):
    b = Batch(0, tile_tets=128)
    first = {}
    for mesh, i, par, contacts in _batch_cells(case, seed):
        c = b.add_cell_like(first[i]) if i in first else b.add_cell(mesh.points, mesh.tets)
        first.setdefault(i, c)
        b.set_viscoplastic(c, par)
        for q in contacts:
            b.add_contact(c, q["kind"], q["k"], q["radius"], q["p0"], q["v"], q["tmove"])
        b.set_integrator(c, 0.01, False)
    b.set_record(1, max(case["steps"], 20), 1024)
    b.finalize()
    return {"case": case, "batch": b}


def _run_batch(state):
    case, b = state["case"], state["batch"]
    b.step(case["steps"])
    out = {"force": b.indenter_force(1).astype(np.float32)}
    if case["points"]:
        out["points"] = [b.points(c) for c in range(case["cells"])]
    return out


# ------------------------------------------------------------------------------------------
# networks
# ------------------------------------------------------------------------------------------
N_IN = 6
GAIN = (0, 1.6)  # exp(1.6 u_0): the surrogate's output gain on its first input
TRAIN = dict(lr=2e-3, lr_min=1e-5, weight_decay=1e-5)
FIT_LR = 2e-2
FREE = np.array([True, True, True, True, True, False])


def _net_inputs(case: dict, seed: int):
    """(parameters, x, target, weight, start) — He-initialised layers, inputs over the unit box,
    smooth curves of them as targets, each weighted by its squared norm (the relative error)."""
    rng = np.random.default_rng([seed, 3])
    fan = [N_IN] + [case["width"]] * case["depth"] + [case["n_out"]]
    par = np.concatenate([np.concatenate([rng.normal(0.0, math.sqrt(2.0 / i), o * i), rng.normal(0.0, 0.02, o)])
                          for i, o in zip(fan[:-1], fan[1:])]).astype(np.float32)
    n = case["rows"]
    x = rng.uniform(-1.0, 1.0, (n, N_IN)).astype(np.float32)
    d = np.linspace(0.05, 1.0, case["n_out"])
    t = np.exp(GAIN[1] * x[:, :1]) * d ** (1.5 + 0.4 * x[:, 1:2]) * (1.0 + 0.2 * np.sin(3.0 * x[:, 2:3] * d + x[:, 3:4]))
    t = t.astype(np.float32)
    w = (1.0 / (t.astype(np.float64) ** 2).sum(1)).astype(np.float32)
    start = rng.uniform(-0.9, 0.9, (n, N_IN)).astype(np.float32)
    start[:, 5] = x[:, 5]
    return par, x, t, w, start


def _prepare_net(case: dict, seed: int):
    par, x, t, w, start = _net_inputs(case, seed)
    m = MLP(N_IN, case["width"], case["depth"], case["n_out"], max_batch=case.get("max_batch", case.get("batch")))
    m.set_params(par)
    m.set_output_gain(*GAIN)
    return {"case": case, "net": m, "x": x, "t": t, "w": w, "start": start, "seed": seed}


def _run_net(state):
    case, m = state["case"], state["net"]
    if case["op"] == "forward":
        return m.forward(state["x"])
    if case["op"] == "backward":
        loss, dx = m.backward(state["x"], state["t"], state["w"], scale=1.0 / case["rows"], want_dx=True)
        return {"loss": loss, "dx": dx, "grads": m.grads()}
    if case["op"] == "train":
        losses = m.train(state["x"], state["t"], steps=case["steps"], batch=case["batch"], weight=state["w"],
                         seed=state["seed"], **TRAIN)
        return {"losses": losses, "params": m.params()}
    x, loss = m.fit_inputs(state["start"], state["t"], FREE, -np.ones(N_IN, np.float32), np.ones(N_IN, np.float32),
                           steps=case["steps"], lr=FIT_LR, weight=state["w"])
    return {"x": x, "loss": loss}


# ------------------------------------------------------------------------------------------
# entry points
# ------------------------------------------------------------------------------------------
def prepare(case: dict, seed: int):
    if case["kind"] == "cell":
        return _prepare_cell(case, seed)
    if case["kind"] == "batch":
        return _prepare_batch(case, seed)
    return _prepare_net(case, seed)


def run(state):
    kind = state["case"]["kind"]
    if kind == "cell":
        return _run_cell(state)
    if kind == "batch":
        return _run_batch(state)
    return _run_net(state)


def _step_work(nt: int, nodes: int, vp: bool) -> tuple[float, float]:
    """Bytes and operations of one step: per tetra the connectivity (16 B), the inverse reference
    shape and volume (40 B) and the viscoplastic state read and written (80 B); per node position,
    velocity and previous force read and written (72 B)."""
    return (136.0 if vp else 56.0) * nt + 72.0 * nodes, (609.0 if vp else 330.0) * nt + 40.0 * nodes


def work(case: dict) -> dict:
    if case["kind"] == "cell":
        _, nt, nodes = mesh_counts(case["radius"])
        b, f = _step_work(nt, nodes, case["material"] == "vp")
        return {"bytes": case["steps"] * b + 24.0 * nodes + (16.0 * nt if case["fields"] else 0.0),
                "flops": case["steps"] * f}
    if case["kind"] == "batch":
        nt = nodes = 0
        for mesh, *_ in _batch_cells(case, 0):
            nt += mesh.num_tetra
            nodes += mesh.num_points
        b, f = _step_work(nt, nodes, True)
        return {"bytes": case["steps"] * b + 8.0 * case["cells"] + (24.0 * nodes if case["points"] else 0.0),
                "flops": case["steps"] * f}
    w, d, o = case["width"], case["depth"], case["n_out"]
    weights = N_IN * w + (d - 1) * w * w + w * o
    params = weights + d * w + o
    rows = case.get("batch", case["rows"])
    row_bytes = 4.0 * (N_IN + o)
    if case["op"] == "forward":
        return {"bytes": 4.0 * params + rows * row_bytes, "flops": 2.0 * weights * rows}
    if case["op"] == "backward":
        return {"bytes": 8.0 * params + rows * (row_bytes + 4.0 * (N_IN + 2)), "flops": 6.0 * weights * rows}
    if case["op"] == "train":  # parameters and both moments read and written, every step
        return {"bytes": case["steps"] * (24.0 * params + rows * row_bytes), "flops": case["steps"] * 6.0 * weights * rows}
    # fitting: the weights once, the rows' inputs and moments stay with their rows
    return {"bytes": 4.0 * params + rows * (row_bytes + 4.0 * (2 * N_IN + 2)), "flops": case["steps"] * 4.0 * weights * rows}


# ------------------------------------------------------------------------------------------
# the same results in 64 bits
# ------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _mm(a, b):
    """Products of 3 x 3 matrices stored [3, 3, n]."""
    return (a[:, :, None] * b[None]).sum(1)


def _tp(a):
    return a.transpose(0, 1)


def _adj(m):
    """Adjugates (transposed cofactors) of [3, 3, n]."""
    return torch.stack([
        torch.stack([m[1, 1] * m[2, 2] - m[1, 2] * m[2, 1], m[0, 2] * m[2, 1] - m[0, 1] * m[2, 2], m[0, 1] * m[1, 2] - m[0, 2] * m[1, 1]]),
        torch.stack([m[1, 2] * m[2, 0] - m[1, 0] * m[2, 2], m[0, 0] * m[2, 2] - m[0, 2] * m[2, 0], m[0, 2] * m[1, 0] - m[0, 0] * m[1, 2]]),
        torch.stack([m[1, 0] * m[2, 1] - m[1, 1] * m[2, 0], m[0, 1] * m[2, 0] - m[0, 0] * m[2, 1], m[0, 0] * m[1, 1] - m[0, 1] * m[1, 0]])])


def _det(m, a):
    return m[0, 0] * a[0, 0] + m[0, 1] * a[1, 0] + m[0, 2] * a[2, 0]


def _tr(m):
    return m[0, 0] + m[1, 1] + m[2, 2]


class _Exact:
    """The explicit step in 64 bits: cells side by side in one set of arrays (node axis last)."""

    def __init__(self, points, tets, model, par, integrator):
        dev = _device()
        self.X = torch.from_numpy(np.ascontiguousarray(points.T)).to(dev)  # [3, np]
        self.tets = torch.from_numpy(np.ascontiguousarray(tets.T)).to(dev)  # [4, nt]
        self.model, self.par, self.integrator = model, par, integrator
        self.I = torch.eye(3, dtype=torch.float64, device=dev)[:, :, None]
        Dm = self.edges(self.X)
        A = _adj(Dm)
        det = _det(Dm, A)
        self.Dmi, self.V0 = A / det, det / 6.0
        self.Fp = self.I.expand(3, 3, self.tets.shape[1]).clone() if model == "vp" else None
        self.eps = torch.zeros_like(self.V0)
        self.x, self.v, self.fo = self.X.clone(), torch.zeros_like(self.X), torch.zeros_like(self.X)
        mass = torch.zeros(self.X.shape[1], dtype=torch.float64, device=dev)
        for k in range(4):
            mass.index_add_(0, self.tets[k], 0.25 * self.V0)
        self.minv = 1.0 / mass
        self.vm = self.p = None

    def edges(self, x):
        return torch.stack([x[:, self.tets[k]] - x[:, self.tets[0]] for k in (1, 2, 3)], 1)

    def mooney(self, B, J, mu1, mu2, kappa):
        t = _tr(B)
        s = mu1 * J ** (-5.0 / 3.0) * (B - t / 3.0 * self.I) + kappa * (J - 1.0) * self.I
        B2 = _mm(B, B)
        return s + mu2 * J ** (-7.0 / 3.0) * (t * B - B2 + (_tr(B2) - t * t) / 3.0 * self.I)

    def element_force(self):
        F = _mm(self.edges(self.x), self.Dmi)
        adjF = _adj(F)
        J = _det(F, adjF)
        q = self.par
        if self.model == "mr":
            g = _mm(adjF, self.mooney(_mm(F, _tp(F)), J, *q))
            w = -self.V0
        elif self.model == "vp":
            adjP = _adj(self.Fp)
            Fe = _mm(F, adjP / _det(self.Fp, adjP))
            Je = _det(Fe, _adj(Fe)).abs()
            s = self.mooney(_mm(Fe, _tp(Fe)), Je, q[0], q[1], q[2])
            g = _mm(adjF, s)
            w = -self.V0.abs() * torch.where(J >= 0, 1.0, -1.0)
            self.p = _tr(s) / 3.0
            dev = s - self.p * self.I
            self.vm = (1.5 * (dev * dev).sum((0, 1))).sqrt()
            rate = q[5] * (self.vm / q[4]) ** q[3]  # no hardening: the yield stress is constant
            Dp = torch.where(self.vm > 0, 1.5 * rate / self.vm.clamp_min(1e-300), torch.zeros_like(rate)) * dev
            self.Fp = self.Fp + _mm(_mm(self.Fp, adjF / J), _mm(Dp, F))
            self.eps = self.eps + rate
        else:
            mu, kp = q
            B = _mm(F, _tp(F))
            if self.model == "svk":
                g = _mm(_tp(F), kp * (_tr(B) - 3.0) * self.I + (B - self.I))
            else:
                Y = B
                for _ in range(10):  # Newton's iteration for the orthogonal polar factor
                    T = _tp(Y)
                    A = _adj(T)
                    Y = 0.5 * (Y + A / _det(T, A))
                S = _mm(_tp(Y), B)
                A = _adj(S)
                g = _mm(self.I + (kp * (_tr(S) - 3.0) - 1.0) * A / _det(S, A), _tp(F))
            w = -self.V0 * mu
        f = _mm(self.Dmi * w, g)  # row k: the force on corner k + 1
        out = torch.zeros_like(self.x)
        out.index_add_(1, self.tets[0], -f.sum(0))
        for k in range(3):
            out.index_add_(1, self.tets[k + 1], f[k])
        return out

    def sphere_integral(self, c, w):
        x = torch.stack([self.x[:, self.tets[k]] for k in range(4)])  # [4, 3, nt]
        d = x.clone()
        d[:, 1] -= w
        e = x[:3] - x[3]
        vol = 0.25 * _det(e, _adj(e)).abs()
        al, be = 0.58541020, 0.13819669
        F = torch.zeros_like(x)
        for g in range(4):
            N = [al if g == k else be for k in range(3)]
            N.append(1.0 - sum(N))
            r = sum(N[k] * d[k] for k in range(4))
            n = r.square().sum(0).sqrt()
            mag = torch.exp(-c["k"] * (n - c["radius"])) / n
            for k in range(4):
                F[k] += mag * N[k] * r
        F = F * vol
        out = torch.zeros_like(self.x)
        for k in range(4):
            out.index_add_(1, self.tets[k], F[k])
        return out

    def contact(self, c, t):
        """Force of one contact (its numbers scalars, or tensors over the nodes) at time t."""
        w = c["p0"] - c["v"] * min(float(t), c["tmove"])
        if c["kind"] == SPHERE_INTEGRAL:
            return self.sphere_integral(c, w)
        f = torch.zeros_like(self.x)
        if c["kind"] == CONTACT_SUBSTRATE:
            f[1] = c["k"] * (w - self.x[1]).clamp_min(0.0)
        elif c["kind"] == CONTACT_PLANE:
            f[1] = -c["k"] * (self.x[1] - w).clamp_min(0.0)
        else:
            r = self.x.clone()
            r[1] -= w
            n = r.square().sum(0).sqrt()
            f = c["k"] * (c["radius"] - n).clamp_min(0.0) * r / n.clamp_min(1e-300)
        return f

    def steps(self, n, contacts, xi):
        for t in range(n):
            f = self.element_force()
            for c in contacts:
                f = f + self.contact(c, t)
            if self.integrator == "vv2":
                a = f * self.minv
                self.v = (self.v + 0.5 * (self.fo + a)) / (1.0 + 0.5 * xi)
                self.fo = a - xi * self.v
                self.x = self.x + self.v + 0.5 * self.fo
            else:
                self.v = (self.v * (1.0 - 0.5 * xi) + 0.5 * (f + self.fo)) / (1.0 + 0.5 * xi)
                self.x = self.x + self.v * (1.0 - 0.5 * xi) + 0.5 * f
                self.fo = f


def _exact_cell(case: dict, seed: int):
    mesh, x, v, fp, contacts = _cell_state(case, seed)
    if case["material"] == "vp":
        model, par = "vp", _cell_workload(case).vp_params()
    else:
        _, E, nu, mr = _elastic(case["material"])
        mu = E / (2.0 * (1.0 + nu))
        if case["material"] in ("svk", "svkk"):
            model, par = case["material"], (mu, nu / (1.0 - 2.0 * nu))
        else:
            model, par = "mr", (mr * mu, (1.0 - mr) * mu, E / (3.0 * (1.0 - 2.0 * nu)))
    e = _Exact(mesh.points, mesh.tets, model, par, case["integrator"])
    e.x = torch.from_numpy(np.ascontiguousarray(x.T)).to(e.x.device)
    e.v = torch.from_numpy(np.ascontiguousarray(v.T)).to(e.x.device)
    if fp is not None:
        e.Fp = torch.from_numpy(fp.reshape(3, 3, -1)).to(e.x.device)
    n = case["steps"]
    e.steps(n, contacts, 0.05 if case["integrator"] == "vv2" else 0.01)
    out = {"force": -e.contact(contacts[1], n)[1].sum().item(), "points": e.x.reshape(-1)}
    if case["fields"]:  # the fields of the last step whose end is an output time
        every = max(n, 20)
        out["von_mises"] = e.vm if n % every == 0 else None
        out["pressure"] = e.p if n % every == 0 else None
    return out


def _exact_batch(case: dict, seed: int):
    cells = _batch_cells(case, seed)
    base, pts, tets, par, nodes = 0, [], [], [], []
    for mesh, _, q, _ in cells:
        pts.append(mesh.points)
        tets.append(mesh.tets + base)
        par.append(np.repeat(np.array(q)[:, None], mesh.num_tetra, 1))
        nodes.append(mesh.num_points)
        base += mesh.num_points
    dev = _device()
    par = torch.from_numpy(np.concatenate(par, 1)).to(dev)
    e = _Exact(np.concatenate(pts), np.concatenate(tets), "vp", tuple(par), "vv")
    owner = torch.from_numpy(np.repeat(np.arange(len(cells)), nodes)).to(dev)
    contacts = []
    for k in range(2):
        c = [q[3][k] for q in cells]
        per = {a: torch.tensor([d[a] for d in c], dtype=torch.float64, device=dev)[owner] for a in ("radius", "p0")}
        contacts.append(dict(kind=c[0]["kind"], k=c[0]["k"], v=c[0]["v"], tmove=c[0]["tmove"], **per))
    n = case["steps"]
    e.steps(n, contacts, 0.01)
    force = torch.zeros(len(cells), dtype=torch.float64, device=dev)
    force.index_add_(0, owner, -e.contact(contacts[1], n)[1])
    out = {"force": force}
    if case["points"]:
        out["points"] = [x.T for x in e.x.split(nodes, 1)]
    return out


class _ExactNet:
    """The network in 64 bits; its parameters as tensors that autograd follows."""

    def __init__(self, case: dict, par):
        fan = [N_IN] + [case["width"]] * case["depth"] + [case["n_out"]]
        p = torch.from_numpy(par.astype(np.float64)).to(_device())
        self.p, pos = [], 0
        for i, o in zip(fan[:-1], fan[1:]):
            self.p += [p[pos:pos + o * i].reshape(o, i).clone().requires_grad_(),
                       p[pos + o * i:pos + o * i + o].clone().requires_grad_()]
            pos += o * i + o

    def __call__(self, x):
        a = x
        for k in range(0, len(self.p), 2):
            a = a @ self.p[k].T + self.p[k + 1]
            if k + 2 < len(self.p):
                a = torch.nn.functional.silu(a)
        return torch.exp(GAIN[1] * x[:, GAIN[0]:GAIN[0] + 1]) * a

    def loss(self, x, t, w):
        return w * (self(x) - t).square().sum(1)

    def flat(self, ts):
        return torch.cat([t.detach().reshape(-1) for t in ts])


def _pcg_rows(n: int, count: int, seed: int) -> np.ndarray:
    """The row order of a training call: a PCG32 stream shuffles every epoch (Fisher-Yates)."""
    M64 = (1 << 64) - 1
    state = (seed * 6364136223846793005 + 1442695040888963407) & M64
    perm, out = list(range(n)), []
    while len(out) < count:
        for k in range(n - 1, 0, -1):
            old = state
            state = (old * 6364136223846793005 + 1442695040888963407) & M64
            xs, rot = (((old >> 18) ^ old) >> 27) & 0xFFFFFFFF, old >> 59
            j = (((xs >> rot) | (xs << ((32 - rot) & 31))) & 0xFFFFFFFF) % (k + 1)
            perm[k], perm[j] = perm[j], perm[k]
        out += perm
    return np.array(out[:count])


def _exact_net(case: dict, seed: int):
    par, x, t, w, start = _net_inputs(case, seed)
    net = _ExactNet(case, par)
    X, T, W = (torch.from_numpy(a.astype(np.float64)).to(_device()) for a in (x, t, w))
    if case["op"] == "forward":
        return net(X).detach()
    if case["op"] == "backward":
        X.requires_grad_()
        loss = net.loss(X, T, W)
        g = torch.autograd.grad(loss.sum() / case["rows"], [X] + net.p)
        return {"loss": loss.detach(), "dx": g[0], "grads": net.flat(g[1:])}
    if case["op"] == "train":
        n, B = case["steps"], case["batch"]
        rows = torch.from_numpy(_pcg_rows(case["rows"], n * B, seed)).to(_device()).reshape(n, B)
        m1, m2 = [torch.zeros_like(p) for p in net.p], [torch.zeros_like(p) for p in net.p]
        losses = []
        for s in range(n):
            loss = net.loss(X[rows[s]], T[rows[s]], W[rows[s]]).mean()
            losses.append(loss.item())
            g = torch.autograd.grad(loss, net.p)
            frac = s / (n - 1) if n > 1 else 0.0
            lr = TRAIN["lr_min"] + 0.5 * (TRAIN["lr"] - TRAIN["lr_min"]) * (1.0 + math.cos(math.pi * frac))
            with torch.no_grad():
                for k, p in enumerate(net.p):
                    m1[k] = 0.9 * m1[k] + 0.1 * g[k]
                    m2[k] = 0.999 * m2[k] + 0.001 * g[k] ** 2
                    if k % 2 == 0:
                        p *= 1.0 - lr * TRAIN["weight_decay"]
                    p -= lr * (m1[k] / (1.0 - 0.9 ** (s + 1))) / ((m2[k] / (1.0 - 0.999 ** (s + 1))).sqrt() + 1e-8)
        return {"losses": np.array(losses), "params": net.flat(net.p)}
    # Fitting: the rows end wherever their valley is flat, and there the descent's last digits
    # decide; only the inputs after a short descent have a value to compare with.
    if case["steps"] > 100:
        return None
    u = torch.from_numpy(start.astype(np.float64)).to(_device())
    free = torch.from_numpy(FREE).to(u.device)
    m1, m2 = torch.zeros_like(u), torch.zeros_like(u)
    for s in range(case["steps"]):
        u.requires_grad_()
        g = torch.autograd.grad(net.loss(u, T, W).sum(), u)[0]
        u = u.detach()
        m1, m2 = 0.9 * m1 + 0.1 * g, 0.999 * m2 + 0.001 * g * g
        step = FIT_LR * (m1 / (1.0 - 0.9 ** (s + 1))) / ((m2 / (1.0 - 0.999 ** (s + 1))).sqrt() + 1e-8)
        u = torch.where(free, (u - step).clamp(-1.0, 1.0), u)
    return {"x": u, "loss": None}


def exact(case: dict, seed: int):
    if case["kind"] == "cell":
        return _exact_cell(case, seed)
    if case["kind"] == "batch":
        return _exact_batch(case, seed)
    return _exact_net(case, seed)
