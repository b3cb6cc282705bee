"""Workloads of the wave stepper, from the smallest room to the largest, through its public entry
points: forward runs in every precision and stencil, and the gradients a material fit takes.

A case is a room's kind, its sizes, the steps of a call and the precision. ``prepare`` gives what a
program that steps that room has in hand: the laid-out grid (the same for every drive), a solver
handle on the GPU, and the seed's drive (and, for a fit, the seed's measured responses and the
materials of the iteration at hand). ``run`` is one call of such a program. ``exact`` is the same
scheme in plain float64 torch.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from acoustic_spaces_b200 import B200WaveSolver, fit, layouts

SPEED = 343.0
STEPS = ((-1, 0, 0), (1, 0, 0), (0, -1, 0), (0, 1, 0), (0, 0, -1), (0, 0, 1),
         (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 1, 0), (-1, 0, -1), (1, 0, -1),
         (-1, 0, 1), (1, 0, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1), (0, 1, 1))  # fmt: skip
TABLES = tuple(f"{kind}{face}_{axis}" for kind in ("keep", "push") for axis in "xyz" for face in ("", "_face"))


def listed() -> list[dict]:
    return [
        # A vocal booth at the low octave bands in one short call, where launches are most of the
        # time: 2,000 cells, resonant walls.
        {"name": "booth", "kind": "box", "x": 2.4, "y": 2.0, "z": 2.2, "cell": 0.18, "speed": 0.0, "branches": 2,
         "receivers": 2, "steps": 128, "precision": "fp32"},
        # A studio of 10,000 cells at the 125 Hz band over a whole response (1,016 steps), the state read
        # after it (to save it and go on later).
        {"name": "studio", "kind": "box", "x": 5.6, "y": 4.5, "z": 3.1, "cell": 0.2, "speed": 0.0, "branches": 2,
         "receivers": 8, "steps": 1016, "precision": "fp32", "state": True},
        # The plain 6 x 4 x 3 m box at 5 cm in double, with its uniform speed ratio.
        {"name": "shoebox_fp64", "kind": "box", "x": 6.0, "y": 4.0, "z": 3.0, "cell": 0.05, "speed": 0.99, "branches": 0,
         "receivers": 1, "steps": 1000, "precision": "fp64"},
        # A closed hall with the 19-point stencil and resonant walls, 869,000 cells.
        {"name": "hall_wide", "kind": "wide", "nx": 151, "ny": 97, "nz": 59, "branches": 3, "receivers": 6, "steps": 600,
         "precision": "fp32"},
        # An auditorium with fitted walls, open through one face into the matched layer, 1.3
        # million cells over 1,016 steps.
        {"name": "auditorium", "kind": "room", "cell": 0.13, "walls": "fitted", "receivers": 16, "steps": 1016,
         "precision": "fp32"},
        # One iteration of a material fit in double on a small room.
        {"name": "fit_fp64", "kind": "fit", "x": 5.0, "y": 4.0, "z": 3.0, "cell": 0.1, "receivers": 4, "steps": 300,
         "segment": 75, "precision": "fp64"},
        # One iteration of a material fit on the 10 x 8 x 4 m room at 5 cm.
        {"name": "fit", "kind": "fit", "x": 10.0, "y": 8.0, "z": 4.0, "cell": 0.05, "receivers": 4, "steps": 500,
         "segment": 250, "precision": "fp32"},
        # The gradient in the walls and in the matched layer's tables, with checkpoints, over a run
        # long enough for sound to come back from the layer.
        {"name": "layer_gradient", "kind": "layer_fit", "cell": 0.16, "receivers": 8, "steps": 320, "segment": 80,
         "precision": "fp32"},
        # Outdoor sound behind a barrier: a 12-cell layer on five sides, porous ground.
        {"name": "outdoor", "kind": "outdoor", "nx": 640, "ny": 176, "nz": 150, "receivers": 64, "steps": 300,
         "precision": "fp32"},
        # A batch: rooms of several sources each, all stepped as one grid.
        {"name": "batch", "kind": "batch", "rooms": 4, "sources": 4, "low": 3.0, "high": 6.0, "receivers": 4,
         "steps": 300, "precision": "fp32"},
        # A long run's compensated precision on the polyhedral room at 6 cm.
        {"name": "room_compensated", "kind": "room", "cell": 0.06, "walls": "fitted", "receivers": 16, "steps": 300,
         "precision": "fp32c"},
        # The polyhedral room at 4 cm (500 x 375 x 250 cells) with fitted walls: the largest grid.
        {"name": "room", "kind": "room", "cell": 0.04, "walls": "fitted", "receivers": 16, "steps": 400,
         "precision": "fp32"},
    ]  # fmt: skip


def _log(rng, low, high):
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def draw(rng) -> dict:
    """One more room of the same kinds: sizes log-uniform from a booth to tens of millions of cells."""
    kind = rng.choice(["box", "box", "wide", "room", "room", "outdoor", "batch", "fit", "layer_fit"])
    precision = rng.choice(["fp32", "fp32", "fp32", "fp64", "fp32c"])
    receivers = rng.choice([1, 2, 3, 5, 8, 16, 33])
    steps = int(_log(rng, 100, 400)) | rng.randrange(2)
    if kind == "box":
        cell, cells = _log(rng, 0.035, 0.2), [_log(rng, 14, top) for top in (160, 130, 90)]
        return {"kind": kind, **{k: round(cell * v, 3) for k, v in zip("xyz", cells)}, "cell": round(cell, 4),
                "speed": rng.choice([0.0, 0.0, 0.97]), "branches": rng.choice([0, 1, 3]), "receivers": receivers,
                "steps": 2 * steps, "precision": precision, "state": math.prod(cells) < 20000}
    if kind == "wide":
        return {"kind": kind, "nx": int(_log(rng, 20, 240)), "ny": int(_log(rng, 20, 160)), "nz": int(_log(rng, 16, 100)),
                "branches": rng.choice([0, 2, 5]), "receivers": receivers, "steps": 2 * steps, "precision": precision}
    if kind == "room":
        return {"kind": kind, "cell": round(_log(rng, 0.06, 0.25), 4), "walls": rng.choice(["fitted", "faces"]),
                "receivers": receivers, "steps": steps, "precision": precision}
    if kind == "outdoor":
        return {"kind": kind, "nx": int(_log(rng, 240, 600)), "ny": int(_log(rng, 96, 200)), "nz": int(_log(rng, 80, 160)),
                "receivers": max(8, receivers), "steps": 300 + steps // 4, "precision": precision}
    if kind == "batch":
        return {"kind": kind, "rooms": rng.randint(2, 5), "sources": rng.randint(1, 4), "low": 2.5,
                "high": round(rng.uniform(3.5, 6.0), 2), "receivers": min(8, receivers), "steps": steps, "precision": precision}
    precision = "fp64" if precision == "fp64" else "fp32"  # (the compensated form has no gradient)
    if kind == "fit":
        cell = _log(rng, 0.06, 0.15)
        return {"kind": kind, "x": round(rng.uniform(3.5, 9.0), 2), "y": round(rng.uniform(3.0, 7.0), 2),
                "z": round(rng.uniform(2.5, 4.0), 2), "cell": round(cell, 4), "receivers": min(8, receivers), "steps": steps,
                "segment": rng.randint(40, 250), "precision": precision}
    cell = _log(rng, 0.16, 0.3)
    return {"kind": kind, "cell": round(cell, 4), "receivers": receivers, "steps": int(52.0 / cell) | rng.randrange(2),
            "segment": rng.randint(30, 120), "precision": precision}


# ---- the rooms ---------------------------------------------------------------------------------


def _resonant(rng, count: int, rate: float) -> layouts.Material:
    """A wall: a real admittance and ``count`` resonant branches spread over the low bands."""
    rows = [layouts.resonant_branch(rng.uniform(0.005, 0.3), rng.uniform(0.5, 8.0), f, rate)
            for f in np.geomspace(30.0, 300.0, count) * rng.uniform(0.8, 1.25, count)]  # fmt: skip
    return layouts.Material(float(rng.uniform(0.02, 0.1)), np.vstack(rows) if rows else np.zeros((0, 3)))


def _box(case) -> tuple[dict, float]:
    rng = np.random.default_rng(11)
    size, cell = np.array([case["x"], case["y"], case["z"]]), case["cell"]
    speed = case["speed"] or None
    rate = SPEED / ((speed or 1.0) * layouts.COURANT * cell)
    room = layouts.shoebox(size, [_resonant(rng, case["branches"], rate) for _ in range(6)])
    clear = min(0.5, 3.2 * cell)
    points = layouts.inside_points(rng, room, size, 1 + case["receivers"], clear, apart=4 * cell)
    built = layouts.cell_face_layout(room, layouts.room_grid(size, cell), points[0], points[1:], speed=speed, rate=rate)
    return built.layout, rate


def _wide(case) -> tuple[dict, float]:
    """A closed box of nx x ny x nz air cells with the isotropic 19-point stencil: weights 1/4 and
    1/8; at a wall the links through it fold back onto the cell's other links (a mirror), and each
    wall met takes the admittance weight 3/4 / (2 L), L the Courant number sqrt(3/4)."""
    rng = np.random.default_rng(12)
    dims = np.array([case["nx"], case["ny"], case["nz"]], np.int64)
    shape = dims + 4
    courant = math.sqrt(0.75)
    rate = SPEED / (courant * 0.1)
    n, sy, sz = int(np.prod(shape)), int(shape[0]), int(shape[0] * shape[1])
    types = np.zeros(tuple(shape[::-1]), np.uint8)
    types[2:-2, 2:-2, 2:-2] = 1
    types = types.reshape(-1)
    inside = np.flatnonzero(types)

    def coords(cells):
        return np.stack([cells % sy, (cells // sy) % int(shape[1]), cells // sz], 1)

    c = coords(inside)
    boundary = inside[((c == 2) | (c == shape - 3)).any(1)]
    probes = layouts.Grid(np.zeros(3), 1.0, tuple(int(v) for v in shape))
    points = rng.uniform(np.full(3, 5.5), shape - 5.5, (1 + case["receivers"], 3))
    for k in range(1, len(points)):
        while np.linalg.norm(points[k] - points[0]) < 4.0:
            points[k] = rng.uniform(np.full(3, 5.5), shape - 5.5)
    fed = layouts.cubic_cells(probes, points[0])
    extra = np.array([i for i, _ in fed if i not in set(boundary.tolist())], np.int64)
    special = np.concatenate([boundary, extra])
    c = coords(special)
    low, high = c == 2, c == shape - 3  # the walls each row's cell meets
    weight = np.zeros((len(special), 18))
    for d, step in enumerate(STEPS):
        gone = [np.where(s < 0, low[:, a], high[:, a]) if s else np.zeros(len(special), bool) for a, s in enumerate(step)]
        rest = np.array(step)[None, :] * ~np.stack(gone, 1)
        for target, to in enumerate(STEPS):
            hit = (rest == np.array(to)).all(1)
            weight[hit, target] += 0.25 if d < 6 else 0.125
    mats = [_resonant(rng, case["branches"], rate) for _ in range(6)]
    per_wall = 0.75 / (2.0 * courant)
    g = np.zeros(len(special))
    states, branch, now, before, gain = [[] for _ in range(len(special))], [], [], [], []
    for wall in range(6):
        rows = np.flatnonzero((low if wall % 2 == 0 else high)[:, wall // 2])
        g[rows] += per_wall * mats[wall].beta
        for m, r, q in mats[wall].branches:
            a = m + 0.5 * r + 0.5 * q
            g[rows] += per_wall * 0.5 / a
            for k in rows:
                states[k].append(len(now))
            now.append(2.0 * m / a), before.append((2.0 * m + q) / a), gain.append(0.5 / a)
    for s in states:
        branch.extend(s)
    has = weight > 0.0
    link_weight = layouts.lowered(weight[has])
    total = (weight * has).sum(1)
    source = np.zeros(len(special), np.float32)
    at = {int(i): k for k, i in enumerate(special)}
    for i, w in fed:
        source[at[i]] += np.float32(w)
    types[special] = 2
    weights = layouts.lowered(np.array([0.25] * 6 + [0.125] * 12))
    starts, cells, probe_weights = [0], [], []
    for p in points[1:]:
        for i, w in layouts.cubic_cells(probes, p):
            cells.append(i), probe_weights.append(w)
        starts.append(len(cells))
    f32 = lambda v: np.asarray(v, np.float64).astype(np.float32)  # noqa: E731
    return {
        "shape": shape.astype(np.uint64), "stencil": np.array([19], np.uint64), "weights": weights,
        "centre": f32([2.0 - weights.astype(np.float64).sum()]), "total": f32([weights.astype(np.float64).sum()]),
        "scaled": np.array([0], np.uint64), "scale": f32([]), "layer_scale": f32([]), "types": types, "special": special,
        "link_start": np.concatenate([[0], np.cumsum(has.sum(1))]).astype(np.uint64),
        "link_direction": np.broadcast_to(np.arange(18, dtype=np.uint8), has.shape)[has], "link_weight": link_weight,
        "coef_a": f32(2.0 - total * (1.0 - layouts.MARGIN)), "coef_b": f32(1.0 - g), "coef_inv": f32(1.0 / (1.0 + g)),
        "source": source, "state_start": np.cumsum([0] + [len(s) for s in states]).astype(np.uint64),
        "state_branch": np.array(branch, np.int32), "state_weight": np.full(len(branch), per_wall, np.float32),
        "branch_now": f32(now), "branch_before": f32(before), "branch_gain": f32(gain),
        "layer_cells": np.zeros(0, np.int64), **{t: f32([]) for t in TABLES},
        "probe_start": np.array(starts, np.uint64), "probe_cells": np.array(cells, np.uint64),
        "probe_weights": np.array(probe_weights, np.float64), "flow_mask": np.zeros(0, np.uint8),
    }, rate  # fmt: skip


@functools.lru_cache(maxsize=3)
def _geometry(key):
    """The laid-out room of a case: its layout, its rate and, for a fit, the builder's own record of
    the rows' materials. A program lays its room out once for all its drives."""
    case = dict(key)
    kind = case["kind"]
    if kind == "box":
        return *_box(case), None
    if kind == "wide":
        return *_wide(case), None
    if kind in ("room", "layer_fit"):
        w = layouts.polyhedral_room(7, cell=case["cell"], receivers=case["receivers"], steps=1,
                                    walls=case.get("walls", "faces"))  # fmt: skip
        return w.built.layout, w.built.rate or SPEED / (layouts.COURANT * case["cell"]), None
    if kind == "outdoor":
        w = layouts.outdoor_halfspace(7, shape=(case["nx"], case["ny"], case["nz"]), receivers=case["receivers"], steps=1)
        return w.built.layout, w.built.rate, None
    if kind == "batch":
        b = layouts.batched_rooms(7, rooms=case["rooms"], sources=case["sources"], dims=(case["low"], case["high"]),
                                  receivers=case["receivers"], steps=1)  # fmt: skip
        return b.stacked.layout, b.rate, None
    # A fit: six walls of one relaxation branch each.
    rng = np.random.default_rng(13)
    size, cell = np.array([case["x"], case["y"], case["z"]]), case["cell"]
    rate = SPEED / (layouts.COURANT * cell)
    truth = fit.Relaxation(np.zeros(6), rng.uniform(0.05, 0.5, 6), np.exp(rng.uniform(math.log(50.0), math.log(500.0), 6)))
    walls = [layouts.Material(0.0, fit.relaxation_branch(g, f, rate)) for g, f in zip(truth.conductance, truth.corner_hz)]
    room = layouts.shoebox(size, walls)
    points = layouts.inside_points(rng, room, size, 1 + case["receivers"], 0.5, apart=4 * cell)
    built = layouts.cell_face_layout(room, layouts.room_grid(size, cell), points[0], points[1:], rate=rate)
    return built.layout, rate, (built, truth)


def _room(case):
    keys = ("kind", "x", "y", "z", "nx", "ny", "nz", "cell", "speed", "branches", "receivers", "walls", "rooms", "sources",
            "low", "high")  # fmt: skip
    return _geometry(tuple((k, case[k]) for k in keys if k in case))


# ---- the inputs --------------------------------------------------------------------------------


def _drive(case, seed: int, rate: float) -> np.ndarray:
    """A pulse of the seed's width, level and start: a Ricker wavelet (no net mass in a closed room)."""
    rng = np.random.default_rng([seed, 1])
    steps, width = case["steps"], rng.uniform(3.0, 7.0)
    t = (np.arange(steps) - 6.0 * width - rng.uniform(0.0, 4.0)) / width
    return (rng.uniform(0.3, 2.0) * (1.0 - t * t) * np.exp(-0.5 * t * t)).astype(np.float32)


def _measured(case, seed: int) -> np.ndarray:
    """Responses to fit: each receiver's direct sound and a decaying tail, of the seed."""
    rng = np.random.default_rng([seed, 2])
    steps = case["steps"]
    tail = rng.standard_normal((case["receivers"], steps)) * np.exp(-np.arange(steps) / (0.4 * steps))
    start = rng.uniform(0.08, 0.3, case["receivers"]) * steps
    return 0.02 * np.where(np.arange(steps)[None, :] >= start[:, None], tail, 0.0)


def _materials(case, seed: int, truth):
    """A fit's materials at the iteration at hand: the true ones, each off by the seed's factor."""
    rng = np.random.default_rng([seed, 3])
    return fit.Relaxation.from_vector(truth.beta, truth.vector() * (1.0 + rng.uniform(-0.3, 0.3, len(truth.vector()))))


def prepare(case, seed):
    layout, rate, fitted = _room(case)
    signal = _drive(case, seed, rate)
    if case["kind"] == "fit":
        built, truth = fitted
        problem = fit.AdjointFit(built, signal, _measured(case, seed), rate, truth.beta, case["precision"], case["segment"])
        # The iteration before, which made the fit's solver and its tape.
        problem.loss_and_gradient(_materials(case, seed + 1, truth))
        return {"kind": "fit", "problem": problem, "materials": _materials(case, seed, truth)}
    solver = B200WaveSolver(layout, precision=case["precision"])
    state = {"kind": case["kind"], "solver": solver, "signal": signal, "state": case.get("state", False)}
    if case["kind"] == "layer_fit":
        solver.set_tape(case["segment"])
        state.update(target=_measured(case, seed), segment=case["segment"])
    return state


def run(state):
    if state["kind"] == "fit":
        loss, slopes, gradient = state["problem"].loss_and_gradient(state["materials"], coefficients=True)
        return {"loss": float(loss), "slopes": slopes, "gradient": gradient}
    solver = state["solver"]
    solver.reset()
    series = solver.run(state["signal"])
    if state["state"]:
        return {"series": series, **solver.state()}
    if state["kind"] != "layer_fit":
        return series
    gradient = solver.gradient(state["signal"], 2.0 * (series - state["target"]), segment=state["segment"])
    return {"series": series, "gradient": gradient}


def work(case):
    """A step's bytes at least: two levels read and one written per interior cell, the rows with
    their links and branch states, the matched layer's state; a gradient steps its room twice."""
    layout, _, _ = _room(case)
    types = np.asarray(layout["types"])
    interior = int(np.count_nonzero(types == 1))
    rows, links, states = len(layout["special"]), len(layout["link_direction"]), len(layout["state_branch"])
    layers = len(layout["layer_cells"])
    wide = int(layout["stencil"][0]) == 19
    e = 8 if case["precision"] == "fp64" else 4
    level = 4 if case["precision"] == "fp32c" else 3
    moved = (level * e + (4 if int(layout["scaled"][0]) else 0)) * interior + (3 * e + 28) * rows + 5 * links
    moved += (3 * e + 16) * states + (14 * e + 4) * layers
    flops = (22 if wide else 9) * interior + 8 * rows + 2 * links + 8 * states + 40 * layers
    passes = 2 if case["kind"] in ("fit", "layer_fit") else 1
    return {"bytes": passes * case["steps"] * moved, "flops": passes * case["steps"] * flops}


# ---- the same in 64 bits -----------------------------------------------------------------------


class _Plain:
    """The scheme of one layout in float64 torch, differentiable in the rows' coefficients (``p``:
    coef_b and coef_inv a row; now, before and gain a branch state; the layer's twelve tables)."""

    def __init__(self, layout, device):
        t64 = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=device)  # noqa: E731
        ti = lambda v: torch.as_tensor(np.asarray(v).astype(np.int64), device=device)  # noqa: E731
        self.nx, self.ny, self.nz = (int(v) for v in layout["shape"])
        sy, sz = self.nx, self.nx * self.ny
        self.n = sz * self.nz
        offsets = ti([x + y * sy + z * sz for x, y, z in STEPS])
        weights = np.asarray(layout["weights"], np.float64)
        self.axial, self.diagonal = float(weights[0]), float(weights[6]) if len(weights) > 6 else 0.0
        self.wide = int(layout["stencil"][0]) == 19
        core = (slice(1, -1),) * 3
        types = torch.as_tensor(np.asarray(layout["types"]), device=device).view(self.nz, self.ny, self.nx)
        self.inside = types[core] == 1
        self.centre, self.total, self.scale = float(layout["centre"][0]), float(layout["total"][0]), None
        if int(layout["scaled"][0]):
            self.scale = t64(layout["scale"]).view(self.nz, self.ny, self.nx)[core]
        self.special = ti(layout["special"])
        rows = len(self.special)
        self.rows = rows
        spread = lambda s: ti(np.repeat(np.arange(len(s) - 1), np.diff(np.asarray(s).astype(np.int64))))  # noqa: E731
        self.link_row = spread(layout["link_start"])
        self.link_cell = self.special[self.link_row] + offsets[ti(layout["link_direction"])]
        self.link_weight = t64(layout["link_weight"])
        self.state_row = spread(layout["state_start"])
        self.state_weight, self.coef_a, self.source = (t64(layout[k]) for k in ("state_weight", "coef_a", "source"))
        branch = np.asarray(layout["state_branch"], np.int64)
        self.p = {"coef_b": t64(layout["coef_b"]), "coef_inv": t64(layout["coef_inv"])}
        for name in ("now", "before", "gain"):
            self.p[name] = t64(np.asarray(layout[f"branch_{name}"], np.float64)[branch])
        self.layer = ti(layout["layer_cells"])
        if len(self.layer):
            self.at = (self.layer % self.nx, (self.layer // sy) % self.ny, self.layer // sz)
            self.strides = (1, sy, sz)
            self.layer_scale = t64(layout["layer_scale"]) if self.scale is not None else 1.0
            self.p.update({k: t64(layout[k]) for k in TABLES})
        self.probe_row = spread(layout["probe_start"])
        self.probes = len(layout["probe_start"]) - 1
        self.probe_cells, self.probe_weights = ti(layout["probe_cells"]), t64(layout["probe_weights"])
        self.device = device

    def rest(self):
        zero = lambda n: torch.zeros(n, dtype=torch.float64, device=self.device)  # noqa: E731
        cells = len(self.layer)
        return [zero(self.n), zero(self.n), zero(len(self.state_row)), zero(len(self.state_row))] + [
            zero(cells) for _ in range(9 if cells else 0)]  # fmt: skip

    def steps(self, state, drive):
        """The series of a piece of the run, and the state after it."""
        p = self.p
        a, b, wa, wb, *layer = state
        series = []
        for s in drive:
            series.append(torch.zeros(self.probes, dtype=torch.float64, device=self.device).index_add(
                0, self.probe_row, self.probe_weights * b[self.probe_cells]))
            v = b.view(self.nz, self.ny, self.nx)
            cut = lambda x, y, z: v[1 + z : self.nz - 1 + z, 1 + y : self.ny - 1 + y, 1 + x : self.nx - 1 + x]  # noqa: E731, B023
            sums = sum(cut(*d) for d in STEPS[1:6]) + cut(*STEPS[0])
            here, before = cut(0, 0, 0), a.view(self.nz, self.ny, self.nx)[1:-1, 1:-1, 1:-1]
            spread = self.axial * sums + (self.diagonal * sum(cut(*d) for d in STEPS[6:]) if self.wide else 0.0)
            if self.scale is None:
                air = self.centre * here + spread - before
            else:
                air = (2.0 - self.total * self.scale) * here + self.scale * spread - before
            new = torch.nn.functional.pad(torch.where(self.inside, air, 0.0), (1,) * 6).view(-1)
            links = torch.zeros(self.rows, dtype=torch.float64, device=self.device).index_add(
                0, self.link_row, self.link_weight * b[self.link_cell])
            own = p["now"] * wb - p["before"] * wa
            flow = torch.zeros(self.rows, dtype=torch.float64, device=self.device).index_add(
                0, self.state_row, self.state_weight * own)
            previous = a[self.special]
            rows = (self.coef_a * b[self.special] + links - p["coef_b"] * previous - flow + self.source * float(s)) * p["coef_inv"]
            wn = wa + (rows - previous)[self.state_row] * p["gain"] + own
            new = new.index_put((self.special,), rows)
            if layer:
                here, total, after = b[self.layer], 0.0, []
                for axis, name in enumerate("xyz"):
                    x, st = self.at[axis], self.strides[axis]
                    part, lo, hi = layer[3 * axis : 3 * axis + 3]
                    kf, pf = p[f"keep_face_{name}"], p[f"push_face_{name}"]
                    lo = kf[x] * lo - pf[x] * (here - b[self.layer - st])
                    hi = kf[x + 1] * hi - pf[x + 1] * (b[self.layer + st] - here)
                    part = p[f"keep_{name}"][x] * part - p[f"push_{name}"][x] * self.layer_scale * (hi - lo)
                    total = total + part
                    after += [part, lo, hi]
                layer = after
                new = new.index_put((self.layer,), total)
            a, b, wa, wb = b, new, wb, wn
        return torch.stack(series, 1), [a, b, wa, wb, *layer]

    def run(self, drive):
        with torch.no_grad():
            return self.steps(self.rest(), drive)

    def gradient(self, drive, target, piece):
        """The series, the misfit and its gradient in ``p``, a piece of the run at a time from kept states."""
        starts, state, series = [], self.rest(), []
        with torch.no_grad():
            for k in range(0, len(drive), piece):
                starts.append(state)
                y, state = self.steps(state, drive[k : k + piece])
                series.append(y)
        series = torch.cat(series, 1)
        slope = 2.0 * (series - target)
        names = [k for k, v in self.p.items() if v.numel()]
        sums = {k: torch.zeros_like(v) for k, v in self.p.items()}
        back = [torch.zeros_like(v) for v in state]
        fixed = dict(self.p)
        for m in reversed(range(len(starts))):
            k = m * piece
            self.p = {n: v.clone().requires_grad_(n in names) for n, v in fixed.items()}
            leaves = [v.clone().requires_grad_(True) for v in starts[m]]
            with torch.enable_grad():
                y, end = self.steps(leaves, drive[k : k + piece])
            outs = [(y, slope[:, k : k + piece])] + [(e, g) for e, g in zip(end, back) if e.requires_grad and e.numel()]
            inputs = [v for v in leaves if v.numel()] + [self.p[n] for n in names]
            grads = iter(torch.autograd.grad([o for o, _ in outs], inputs, [g for _, g in outs], allow_unused=True))
            back = [(lambda g, v: torch.zeros_like(v) if g is None else g)(next(grads), v) if v.numel() else v for v in leaves]
            for n in names:
                g = next(grads)
                if g is not None:
                    sums[n] += g
        self.p = fixed
        return series, float(((series - target) ** 2).sum()), sums


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    layout, rate, fitted = _room(case)
    signal = _drive(case, seed, rate)
    if case["kind"] not in ("fit", "layer_fit"):
        series, (a, b, wa, wb, *_) = _Plain(layout, device).run(signal)
        if not case.get("state"):
            return series.cpu()
        return {"series": series.cpu(), "current": b.cpu(), "previous": a.cpu(), "branch_current": wb.cpu(),
                "branch_previous": wa.cpu(), "layer": None}  # fmt: skip
    target = torch.as_tensor(_measured(case, seed), device=device)
    if case["kind"] == "fit":
        built, truth = fitted
        # The iteration's coefficients as the layout holds them (float32), from the materials.
        params, sens = _materials(case, seed, truth), built.sensitivity
        owner = np.asarray(sens["branch_material"], np.int64)
        r = 1.0 / params.conductance[owner]
        q = r * 2.0 * math.pi * params.corner_hz[owner] / rate
        a = 0.5 * (r + q)
        wall = np.zeros(len(params.conductance))
        np.add.at(wall, owner, 0.5 / a)
        g = sens["edge_weight"] * sens["edge_admittance"] + np.bincount(
            sens["row"], sens["weight"] * wall[sens["material"]], minlength=sens["boundary_rows"])
        layout = dict(layout, branch_now=np.zeros(len(a), np.float32), branch_before=(q / a).astype(np.float32),
                      branch_gain=(0.5 / a).astype(np.float32))  # fmt: skip
        for name, value in (("coef_b", 1.0 - sens["r"] * g), ("coef_inv", 1.0 / (1.0 + sens["r"] * g))):
            layout[name] = np.concatenate([value.astype(np.float32), layout[name][len(g):]])
    plain = _Plain(layout, device)
    series, loss, sums = plain.gradient(signal, target, 20)
    gradient = {k: v.cpu() for k, v in sums.items()}
    if case["kind"] == "fit":
        return {"loss": loss, "slopes": None, "gradient": gradient}
    return {"series": series.cpu(), "gradient": gradient}
