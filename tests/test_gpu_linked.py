"""Slabs of small closed rooms, cut through their air into unequal parts and stepped together inside the library
(fdtd_run_linked), against the whole grid to the bit (needs a B200): a plane that a neighbour's copy fills stays what
the copy made it, whichever slab's step ends first."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from acoustic_spaces_b200 import B200WaveSolver, _abi, layouts, slabs
from oracle.oracle import OracleSolver

pytestmark = pytest.mark.gpu


def _box(shape, speed):
    rng = np.random.default_rng(9)
    cell, rate = 0.1, 5000.0
    size = np.asarray(shape, float) * cell
    walls = [layouts.Material(0.05, np.vstack([layouts.resonant_branch(0.1, 2.0, f, rate) for f in rng.uniform(40, 200, 2)]))
             for _ in range(6)]  # fmt: skip
    grid = layouts.Grid(-2.0 * cell * np.ones(3), cell, tuple(int(v) + 4 for v in shape))
    points = [size * np.array([0.5, 0.5, f]) for f in (0.55, 0.12, 0.4, 0.9)]
    return layouts.cell_face_layout(layouts.shoebox(size, walls), grid, points[0], points[1:], speed=speed, rate=rate).layout


def _bounds(layout, shares):
    """Cuts nearest to these shares of the planes, through no probe's cells."""
    nz = int(layout["shape"][2])
    cut = {b for lo, hi in slabs._probe_spans(layout) for b in range(lo + 1, hi + 1)}
    free = [b for b in range(4, nz - 3) if b not in cut]
    at = [0] + [min(free, key=lambda b: abs(b - share * nz)) for share in shares] + [nz]
    assert at == sorted(set(at))
    return list(zip(at[:-1], at[1:]))


def _run(gpus, parts, order, signal):
    """run_linked with the handles listed in `order`."""
    import torch

    lib, place = _abi.load_library(), {slab: k for k, slab in enumerate(order)}
    joined = slabs.links(parts)
    link_array = (_abi.FdtdPlaneLink * len(joined))()
    for k, (a, b, pa, pb) in enumerate(joined):
        link_array[k].from_, link_array[k].to, link_array[k].from_plane, link_array[k].to_plane = place[a], place[b], pa, pb
    listed = [gpus[k] for k in order]
    signals = [torch.from_numpy(signal).cuda() for _ in listed]
    outs = [torch.zeros((max(1, s.probes), len(signal)), dtype=torch.float64, device="cuda") for s in listed]
    torch.cuda.synchronize()
    pointers = ctypes.c_void_p * len(listed)
    status = lib.fdtd_run_linked(pointers(*[s._handle for s in listed]), len(listed), link_array, len(joined),
                                 pointers(*[t.data_ptr() for t in signals]), len(signal),
                                 pointers(*[t.data_ptr() for t in outs]), len(signal))  # fmt: skip
    assert status == _abi.FDTD_OK, lib.fdtd_global_error()
    for s in listed:
        s.synchronize()
    return [outs[place[k]][: gpus[k].probes].cpu().numpy() for k in range(len(gpus))]


@pytest.mark.parametrize("precision", ["fp32", "fp64", "fp32c"])
@pytest.mark.parametrize("shares", [(0.2,), (0.8,), (0.2, 0.7)])
@pytest.mark.parametrize("shape, speed", [((12, 9, 26), None), ((13, 30, 22), 0.95)])
def test_gpu_linked_small_slabs_step_as_the_whole_grid(shape, speed, shares, precision):
    layout = _box(shape, speed)
    parts = [slabs.slab(layout, _bounds(layout, shares), r) for r in range(len(shares) + 1)]
    signal = np.random.default_rng(2).standard_normal(150).astype(np.float32)
    whole = OracleSolver(layout, precision)
    expected = whole.run(signal)
    state = whole.state()["current"]
    gpus = [B200WaveSolver(p.layout, precision=precision, autotune=False) for p in parts]
    plane = int(layout["shape"][0]) * int(layout["shape"][1])
    for order in (list(range(len(gpus))), list(range(len(gpus)))[::-1]):
        for g in gpus:
            g.reset()
        halves = [_run(gpus, parts, order, piece) for piece in (signal[:61], signal[61:])]
        records = [np.concatenate(pair, axis=1) for pair in zip(*halves)]
        assert np.array_equal(slabs.gather_records(parts, records, len(expected), len(signal)), expected)
        for part, g in zip(parts, gpus):
            mine = g.state()["current"][(part.z0 - part.lo) * plane : (part.z1 - part.lo) * plane]
            assert np.array_equal(mine, state[part.z0 * plane : part.z1 * plane])
