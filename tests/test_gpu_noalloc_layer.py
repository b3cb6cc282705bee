"""fdtd_gradient_noalloc on grids with a matched layer (needs a B200): what fits the pool by the layer's cells is taken,
however thin the layer lies over the grid's quads, and gives fdtd_gradient's result."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from acoustic_spaces_b200 import B200WaveSolver, _abi, layouts

pytestmark = pytest.mark.gpu

_F64 = ctypes.POINTER(ctypes.c_double)


def _layered(lone, speed=None):
    """A closed box with layer cells in its air: a block of them, or single cells, each in a quad of its own and with a
    quad of its own below it along every axis (sixteen lanes a cell)."""
    cell = 0.1
    size = np.array([30, 20, 20]) * cell
    walls = [layouts.Material(0.05, np.zeros((0, 3))) for _ in range(6)]
    grid = layouts.Grid(-2.0 * cell * np.ones(3), cell, (34, 24, 24))
    points = [size * 0.5, size * np.array([0.3, 0.4, 0.6])]
    layout = dict(layouts.cell_face_layout(layouts.shoebox(size, walls), grid, points[0], points[1:], speed=speed, rate=5000.0).layout)
    types = np.array(layout["types"], np.uint8).reshape(24, 24, 34)
    chosen = np.zeros(types.shape, bool)
    if lone:
        chosen[4:-3:3, 4:-3:3, 4:-3:8] = True
    else:
        chosen[6:12, 6:12, 5:16] = True
    chosen &= types == 1
    types[chosen] = 3
    layout.update(types=types.reshape(-1), layer_cells=np.flatnonzero(chosen.reshape(-1)).astype(np.int64))
    if speed:
        layout["layer_scale"] = np.asarray(layout["scale"], np.float32)[layout["layer_cells"]].copy()
    push = np.float32(0.95) * np.sqrt(np.float32(np.asarray(layout["weights"]).reshape(-1)[0]))
    for axis, n in zip("xyz", (34, 24, 24)):
        for face in ("", "_face"):
            layout[f"keep{face}_{axis}"] = np.full(n + 1, 0.97, np.float32)
            layout[f"push{face}_{axis}"] = np.full(n + 1, push, np.float32)
    return layout


def _noalloc(solver, signal, dloss, segment):
    info = solver.info()
    out = {k: np.zeros(int(n)) for k, n in (("coef_b", info.special_cells), ("coef_inv", info.special_cells),
                                              ("now", info.branch_states), ("before", info.branch_states),
                                              ("gain", info.branch_states))}  # fmt: skip
    status = _abi.load_library().fdtd_gradient_noalloc(
        solver._handle, signal.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), len(signal), dloss.ctypes.data_as(_F64),
        segment, *(a.ctypes.data_as(_F64) for a in out.values()))  # fmt: skip
    return status, dict(out, **solver.layer_gradient()) if status == _abi.FDTD_OK else None


def _case(layout, precision, steps):
    solver = B200WaveSolver(layout, precision=precision)
    signal = np.random.default_rng(8).standard_normal(steps).astype(np.float32)
    y = solver.run(signal)
    solver.reset()
    return solver, signal, np.ascontiguousarray(y * np.linspace(0.5, 1.5, steps))


def _close(got, expected, precision):
    rtol = 1e-12 if precision == "fp64" else 1e-6
    assert got.keys() == expected.keys()
    for key in expected:
        scale = np.max(np.abs(expected[key])) if expected[key].size else 0.0
        np.testing.assert_allclose(got[key], expected[key], rtol=rtol, atol=rtol * scale, err_msg=key)
    assert np.any(expected["keep_x"]) and np.any(expected["push_face_z"])


@pytest.mark.parametrize("precision, steps", [("fp32", 550), ("fp64", 230)])
def test_gpu_noalloc_takes_layers_of_lone_cells(precision, steps):
    solver, signal, dloss = _case(_layered(True), precision, steps)
    cells = int(solver.info().layer_cells)
    size = 8 if precision == "fp64" else 4
    assert 4 << 20 < 18 * size * cells * steps < 10 << 20  # (by lanes sixteen times as much, past any pool)
    status, got = _noalloc(solver, signal, dloss, 0)
    assert status == _abi.FDTD_OK, _abi.load_library().fdtd_last_error(solver._handle)
    _close(got, solver.gradient(signal, dloss, segment=0), precision)


@pytest.mark.parametrize("speed", [None, 0.95])
@pytest.mark.parametrize("precision, steps, segment", [("fp32", 320, 0), ("fp32", 320, 200), ("fp32", 320, 40),
                                                       ("fp64", 140, 0), ("fp64", 140, 90), ("fp64", 140, 20)])  # fmt: skip
def test_gpu_noalloc_layers_by_cells_and_by_lanes(precision, steps, segment, speed):
    """392 layer cells of 576 lanes: the whole run's factors fit the pool by cells alone, the segments' by lanes too."""
    solver, signal, dloss = _case(_layered(False, speed), precision, steps)
    status, got = _noalloc(solver, signal, dloss, segment)
    assert status == _abi.FDTD_OK, _abi.load_library().fdtd_last_error(solver._handle)
    _close(got, solver.gradient(signal, dloss, segment=segment), precision)
