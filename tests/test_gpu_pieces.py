"""Launched runs that are cut into pieces (the probes' cells are gathered over so many steps at most): what a gradient
records of them is the whole run's (needs a B200)."""

from __future__ import annotations

import numpy as np
import pytest
from conftest import load_golden

from acoustic_spaces_b200 import B200WaveSolver, layouts
from oracle.oracle import OracleSolver

pytestmark = pytest.mark.gpu


def _box():
    rng = np.random.default_rng(5)
    cell, rate = 0.1, 5000.0
    size = np.array([12, 9, 11]) * cell
    walls = [layouts.Material(0.05, layouts.resonant_branch(0.1, 2.0, f, rate)[None]) for f in rng.uniform(40, 200, 6)]
    grid = layouts.Grid(-2.0 * cell * np.ones(3), cell, (16, 13, 15))
    points = [size * 0.5, size * 0.5 + np.array([0.0, 0.0, 0.31 * size[2]])]
    return layouts.cell_face_layout(layouts.shoebox(size, walls), grid, points[0], points[1:], rate=rate).layout


def _repeated(layout, times):
    """The same layout with its probes' cells listed `times` times over (a plane of receivers), its first probes first."""
    starts = np.asarray(layout["probe_start"], np.uint64)
    count = starts[-1]
    tails = [starts[1:] + np.uint64(k) * count for k in range(times)]
    return dict(layout, probe_start=np.concatenate([starts[:1], *tails]), probe_cells=np.tile(layout["probe_cells"], times),
                probe_weights=np.tile(layout["probe_weights"], times))  # fmt: skip


def _gradient(layout, precision, steps, segment, tape, *, tables=True, tangent=None, launched=True):
    solver = B200WaveSolver(layout, precision=precision)
    if launched:
        solver.set_streams(1)  # each step's kernels launched
    if tangent is not None:
        solver.set_layer_tangent(tangent)
    if tape:
        solver.set_tape(segment, layer_tables=tables)
    drive = np.random.default_rng(4).standard_normal(steps).astype(np.float32)
    y = solver.run(drive)
    solver.reset()
    dloss = np.zeros_like(y)
    dloss[0] = y[0] * np.linspace(0.5, 1.5, steps)
    return solver.gradient(drive, dloss, segment=segment, layer_tables=tables)


def _same(a, b):
    assert a.keys() == b.keys()
    for key in a:
        assert np.array_equal(a[key], b[key]), key
        assert np.any(b[key])


@pytest.mark.parametrize("tape", [False, True])
def test_gpu_gradients_of_segments_longer_than_a_piece(tape):
    layout = _box()
    _same(_gradient(layout, "fp32", 1500, 0, tape), _gradient(layout, "fp32", 1500, 300, False))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("tape", [False, True])
def test_gpu_gradients_of_many_receivers(tape, precision):
    """200,000 probe cells: pieces of 40 steps, in double of 20."""
    layout = _box()
    layout = _repeated(layout, 200_000 // len(layout["probe_cells"]))
    _same(_gradient(layout, precision, 150, 100, tape), _gradient(layout, precision, 150, 18, False))


@pytest.mark.parametrize("kind", ["tables", "walls", "tangent"])
@pytest.mark.parametrize("tape", [False, True])
def test_gpu_layer_gradients_of_many_receivers(tape, kind):
    layout = layouts.polyhedral_room(2, cell=0.3, receivers=2, steps=1).built.layout
    layout = _repeated(layout, 200_000 // len(layout["probe_cells"]))
    tangent = layouts.damping_tangent(layout, layouts.LAYER_CELLS, layouts.LAYER_DAMPING) if kind == "tangent" else None
    args = dict(tables=kind == "tables", tangent=tangent)
    a = _gradient(layout, "fp64", 150, 100, tape, **args)
    b = _gradient(layout, "fp64", 150, 18, False, **args)
    if kind != "tangent":
        return _same(a, b)
    # (The tangent's products are added up a segment at a time in the step's own precision.)
    for key in a:
        np.testing.assert_allclose(a[key], b[key], rtol=1e-10, atol=1e-10 * np.abs(b[key]).max(), err_msg=key)


@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp32c"])
@pytest.mark.parametrize("kind", ["box", "wide", "layer"])
def test_gpu_single_steps_between_longer_runs(kind, precision):
    if kind == "box":
        layout = _box()
    elif kind == "wide":
        layout = load_golden("resonant19")[0]
    else:
        layout = layouts.polyhedral_room(2, cell=0.3, receivers=3, steps=1).built.layout
    drive = np.random.default_rng(6).standard_normal(70).astype(np.float32)
    solver, oracle = B200WaveSolver(layout, precision=precision), OracleSolver(layout, precision)
    cuts = [0, 1, 2, 3, 20, 21, 23, 24, 25, 69, 70]
    got = np.concatenate([solver.run(drive[i:j]) for i, j in zip(cuts[:-1], cuts[1:])], axis=1)
    assert np.array_equal(got, oracle.run(drive))
    mine, theirs = solver.state(), oracle.state()
    for key in mine:
        assert np.array_equal(mine[key], theirs[key]), key


@pytest.mark.parametrize("tape", [False, True])
def test_gpu_gradients_of_segments_of_one_step(tape):
    layout = _box()
    args = dict(steps=33, precision="fp32")
    _same(_gradient(layout, segment=1, tape=tape, launched=False, **args), _gradient(layout, segment=33, tape=False, **args))


@pytest.mark.parametrize("cells", [1, 523_000, 540_000])
@pytest.mark.parametrize("launched", [False, True])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_gpu_records_of_many_receivers(cells, launched, precision):
    """Gathered over a launch's steps, over sixteen, or (past 524,288 cells, half as many in double) read every step."""
    layout = _box()
    times = -(-cells // len(layout["probe_cells"]))
    drive = np.random.default_rng(6).standard_normal(70).astype(np.float32)
    solver = B200WaveSolver(_repeated(layout, times), precision=precision)
    if launched:
        solver.set_streams(1)
    assert solver.info().device_bytes < 80e6
    got = np.concatenate([solver.run(drive[:37]), solver.run(drive[37:])], axis=1)
    assert np.array_equal(got, np.tile(OracleSolver(layout, precision).run(drive), (times, 1)))


@pytest.mark.parametrize("speed", [None, 0.97])
def test_gpu_rows_that_shared_memory_does_not_hold(speed):
    """A 7.5M-cell room in double, 1550 rows a block of 5 branch states each: the resident stepper reads its rows' tables
    from memory."""
    rng = np.random.default_rng(7)
    shape = np.array([200, 195, 192])
    walls = [layouts.Material(0.05, np.vstack([layouts.resonant_branch(0.1, 2.0, f, 5000.0) for f in rng.uniform(40, 200, 5)]))
             for _ in range(6)]  # fmt: skip
    grid = layouts.Grid(-0.2 * np.ones(3), 0.1, tuple(int(v) + 4 for v in shape))
    points = [np.array([0.35, 0.35, 0.35]), np.array([0.75, 0.45, 0.35])]
    layout = layouts.cell_face_layout(layouts.shoebox(0.1 * shape, walls), grid, points[0], points[1:], speed=speed,
                                      rate=5000.0).layout  # fmt: skip
    drive = rng.standard_normal(14).astype(np.float32)
    solver, oracle = B200WaveSolver(layout, precision="fp64", autotune=False), OracleSolver(layout, "fp64")
    assert np.array_equal(np.concatenate([solver.run(drive[:9]), solver.run(drive[9:])], axis=1), oracle.run(drive))
    mine, theirs = solver.state(), oracle.state()
    for key in mine:
        assert np.array_equal(mine[key], theirs[key]), key
