"""The resident stepper, the sweep by columns and the matched layer by quads on the sizes where they can go wrong, against
the oracle to the bit (needs a B200): rows that end within a quad or fill the pitch, one column to
many tasks a warp, a cluster or the whole GPU, runs longer than a launch, layers whose cells come in
any order, the layer's state in shared memory or not, and handles stepped from two threads."""

from __future__ import annotations

import threading

import numpy as np
import pytest
from conftest import load_golden

from acoustic_spaces_b200 import B200WaveSolver, layouts
from oracle.oracle import OracleSolver

pytestmark = pytest.mark.gpu


def _box(shape, *, speed=None, branches=2, receivers=2, seed=3):
    """A closed box of shape air cells (two solid cells round it), resonant walls."""
    rng = np.random.default_rng(seed)
    cell, rate = 0.1, 5000.0
    size = np.asarray(shape, float) * cell
    walls = [layouts.Material(0.05, np.vstack([layouts.resonant_branch(0.1, 2.0, f, rate) for f in rng.uniform(40, 200, branches)])
                              if branches else np.zeros((0, 3))) for _ in range(6)]  # fmt: skip
    room = layouts.shoebox(size, walls)
    grid = layouts.Grid(-2.0 * cell * np.ones(3), cell, tuple(int(v) + 4 for v in shape))
    points = [size * 0.5] + [size * 0.5 + np.array([0.0, 0.0, s * 0.31 * size[2]]) for s in (1, -1, 0.9)[:receivers]]
    return layouts.cell_face_layout(room, grid, points[0], points[1:], speed=speed, rate=rate).layout


def _equal(layout, drive, cuts, precision, launched=False):
    gpu, oracle = B200WaveSolver(layout, precision=precision), OracleSolver(layout, precision)
    if launched:
        gpu.set_streams(1)
    a = np.concatenate([gpu.run(drive[i:j]) for i, j in zip(cuts[:-1], cuts[1:])], axis=1)
    assert np.array_equal(a, oracle.run(drive))
    mine, theirs = gpu.state(), oracle.state()
    for key in mine:
        assert np.array_equal(mine[key], theirs[key]), key


def _drive(steps, seed=0):
    return np.random.default_rng(seed).standard_normal(steps).astype(np.float32)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp32c"])
@pytest.mark.parametrize(
    "shape, speed",
    [((12, 9, 11), None), ((13, 16, 13), 0.9), ((28, 12, 14), None), ((60, 61, 10), None), ((77, 50, 47), 0.97), ((140, 90, 61), None)],
)  # (12 + 4 cells fill the pitch of 16; 13 and 77 end within a quad; the last spans several tasks a warp)
@pytest.mark.parametrize("launched", [False, True])
def test_gpu_boxes_of_odd_sizes_step_as_the_oracle_does(shape, speed, precision, launched):
    steps = 90 if np.prod(shape) < 1e5 else 40
    _equal(_box(shape, speed=speed), _drive(steps), [0, 1, 34, steps], precision, launched)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp32c"])
@pytest.mark.parametrize("shape, branches, speed", [((11, 12, 11), 0, None), ((18, 18, 18), 3, 0.95), ((28, 28, 28), 2, None), ((30, 29, 31), 4, None)])
def test_gpu_grids_of_one_cluster_step_as_the_oracle_does(shape, branches, speed, precision):
    """A block's tasks fewer than a warp's, planes a power of two apart, and both sides of the line to the whole GPU;
    the probes written out within a run and at its end."""
    _equal(_box(shape, speed=speed, branches=branches, receivers=1), _drive(203), [0, 1, 66, 203], precision)


def test_gpu_runs_longer_than_a_launch():
    _equal(_box((12, 10, 13)), _drive(2111), [0, 1030, 1031, 2111], "fp32")


@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp32c"])
@pytest.mark.parametrize("count, launched", [(2, False), (9, False), (9, True)])
def test_gpu_wide_grids_step_as_the_oracle_does(count, launched, precision):
    layout, signal, _ = load_golden("resonant19")
    stacked = layouts.stack([layout] * count, across=3).layout
    _equal(stacked, signal[:70], [0, 33, 70], precision, launched)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp32c"])
@pytest.mark.parametrize("cell", [0.3, 0.21, 0.16, 0.13])  # (0.13: in double more state than shared memory holds)
@pytest.mark.parametrize("launched", [False, True])
def test_gpu_layers_step_as_the_oracle_does(cell, precision, launched):
    w = layouts.polyhedral_room(2, cell=cell, receivers=3, steps=1)
    _equal(w.built.layout, _drive(45), [0, 20, 45], precision, launched)


@pytest.mark.parametrize("name", ["open_layer", "open_layer_speed", "fitted_open"])
@pytest.mark.parametrize("launched", [False, True])
def test_gpu_layer_cells_in_any_order(name, launched):
    layout, signal, reference = load_golden(name)
    order = np.random.default_rng(1).permutation(len(layout["layer_cells"]))
    layout = dict(layout, layer_cells=layout["layer_cells"][order])
    if len(layout["layer_scale"]):
        layout["layer_scale"] = layout["layer_scale"][order]
    solver = B200WaveSolver(layout)
    if launched:
        solver.set_launch(2, 3)
    got = np.concatenate([solver.run(signal[:91]), solver.run(signal[91:])], axis=1)
    assert np.array_equal(got, reference)
    oracle = OracleSolver(layout)
    oracle.run(signal)
    assert np.array_equal(solver.state()["layer"], oracle.state()["layer"])


@pytest.mark.parametrize("name", ["resonant7", "fitted_closed", "fitted_open", "speed19"])
def test_gpu_chosen_launches_step_as_the_resident_stepper_does(name):
    layout, signal, reference = load_golden(name)
    solver = B200WaveSolver(layout)
    head = solver.run(signal[:100])
    solver.set_streams(0)  # launched from here on
    assert np.array_equal(np.concatenate([head, solver.run(signal[100:])], axis=1), reference)


def test_gpu_handles_step_from_two_threads():
    cases = [(_box((60, 61, 30), seed=s), _drive(300, s)) for s in (1, 2)]
    alone = [B200WaveSolver(lay).run(d) for lay, d in cases]
    solvers, got = [B200WaveSolver(lay) for lay, _ in cases], [None, None]

    def step(k):
        runs = []
        for _ in range(5):
            solvers[k].reset()
            runs.append(solvers[k].run(cases[k][1]))
        got[k] = runs

    threads = [threading.Thread(target=step, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in (0, 1):
        assert all(np.array_equal(y, alone[k]) for y in got[k])


# ---- the reverse steps -------------------------------------------------------------------------


def _gradients(layout, precision, steps, segment, tape, tables=True, tangent=None, launched=False):
    solver = B200WaveSolver(layout, precision=precision)
    if launched:
        solver.set_adjoint_launch(0, 8)
    if tangent is not None:
        solver.set_layer_tangent(tangent)
    if tape:
        solver.set_tape(segment, layer_tables=tables)
    drive = _drive(steps, 4)
    y = solver.run(drive)
    solver.reset()
    dloss = y * np.linspace(0.5, 1.5, steps)
    return solver.gradient(drive, dloss, segment=segment, layer_tables=tables)


def _same(a, b):
    assert a.keys() == b.keys()
    for key in a:
        assert np.array_equal(a[key], b[key]), key


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("tape", [False, True])
@pytest.mark.parametrize("shape, speed", [((12, 9, 11), None), ((13, 16, 13), 0.9), ((60, 41, 30), None), ((90, 77, 40), 0.97)])
def test_gpu_resident_reverse_steps_equal_the_launched_ones(shape, speed, tape, precision):
    layout = _box(shape, speed=speed)
    args = (layout, precision, 61, 20, tape)
    _same(_gradients(*args), _gradients(*args, launched=True))


@pytest.mark.parametrize("name", ["resonant19", "speed19"])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_gpu_resident_reverse_wide_steps_equal_the_launched_ones(name, precision):
    layout = layouts.stack([load_golden(name)[0]] * 4, across=2).layout
    _same(_gradients(layout, precision, 50, 25, True), _gradients(layout, precision, 50, 25, True, launched=True))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("kind", ["tables", "walls", "tangent"])
@pytest.mark.parametrize("cell", [0.3, 0.2])
def test_gpu_resident_reverse_layers_equal_the_launched_ones(cell, kind, precision):
    layout = layouts.polyhedral_room(2, cell=cell, receivers=3, steps=1).built.layout
    tangent = layouts.damping_tangent(layout, layouts.LAYER_CELLS, layouts.LAYER_DAMPING) if kind == "tangent" else None
    args = (layout, precision, 130, 50, True, kind == "tables", tangent)
    _same(_gradients(*args), _gradients(*args, launched=True))
