"""More sources and receivers than a column's mask has bits (on a GPU): 33 and more points, several in
one cell, in one column and in one chunk, and most columns with none; every scheme bit for bit like the
oracle, and source gradients of the adjoint like those of the same sources a few at a time."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AIR, CudaAcousticFDTD, Grid, RoomBatch, WallAdmittances
from ac_fdtd_b200.adjoint import DifferentiableRoom
from oracle.leapfrog import OracleFDTD

pytestmark = pytest.mark.gpu

SHAPES = [(11, 9, 24), (7, 12, 13)]
WALLS = WallAdmittances(0.4, 0.1, 0.0, 0.7, 0.2, 0.05)


def _points(shape, sources, receivers):
    """Cells: a fifth of the points in one column, some of those in one cell."""
    rng = np.random.default_rng(shape)
    cells = [tuple(int(rng.integers(n)) for n in shape) for _ in range(sources + receivers)]
    column = (shape[1] // 2, shape[2] // 2)
    for n in range(0, len(cells), 5):
        cells[n] = (cells[n][0] if n % 2 else 3, *column)
    signals = rng.standard_normal((sources, 20))
    return cells[:sources], signals, cells[sources:]


def _add(solver, shape, sources, receivers, dx):
    at, signals, heard = _points(shape, sources, receivers)
    for cell, signal in zip(at, signals):
        solver.add_volume_source(tuple((c + 0.5) * dx for c in cell), signal)
    for cell in heard:
        solver.add_pressure_receiver(tuple((c + 0.5) * dx for c in cell))
    return solver


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("sources, receivers", [(1, 31), (1, 32), (40, 7), (3, 150)])
@pytest.mark.parametrize("scheme, steps_per_graph", [("two_sweeps", 64), ("two_sweeps", 0), ("fused", 0)])
def test_recordings_equal_the_oracle(shape, dtype, sources, receivers, scheme, steps_per_graph):
    grid = Grid(dx=0.03, nx=shape[0], ny=shape[1], nz=shape[2])
    solver = CudaAcousticFDTD(grid, dtype=dtype, walls=WALLS, scheme=scheme, steps_per_graph=steps_per_graph)
    oracle = OracleFDTD(grid, AIR, dtype=dtype, walls=WALLS)
    for s in (solver, oracle):
        _add(s, shape, sources, receivers, 0.03)
        s.run(30)
    np.testing.assert_array_equal(solver.recorded_pressure, oracle.recorded_pressure)
    np.testing.assert_array_equal(solver.p, oracle.p)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_a_batch_equals_the_oracle(dtype):
    batch = RoomBatch([dict(grid=Grid(dx=0.03, nx=s[0], ny=s[1], nz=s[2]), walls=WALLS) for s in SHAPES],
                      dtype=dtype, scheme="fused")
    want = []
    for r, shape in enumerate(SHAPES):
        at, signals, heard = _points(shape, 2, 50)
        oracle = _add(OracleFDTD(Grid(dx=0.03, nx=shape[0], ny=shape[1], nz=shape[2]), AIR, dtype=dtype, walls=WALLS),
                      shape, 2, 50, 0.03)
        for cell, signal in zip(at, signals):
            batch.add_volume_source(r, tuple((c + 0.5) * 0.03 for c in cell), signal)
        for cell in heard:
            batch.add_pressure_receiver(r, tuple((c + 0.5) * 0.03 for c in cell))
        oracle.run(30)
        want.append(oracle.recorded_pressure)
    batch.run(30)
    for r in range(len(SHAPES)):
        np.testing.assert_array_equal(batch.recorded_pressure(r), want[r])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SHAPES)
def test_source_gradients(shape, dtype):
    """The adjoint does not depend on how many other sources are listened to."""
    def gradient(sources):
        grid = Grid(dx=0.03, nx=shape[0], ny=shape[1], nz=shape[2])
        room = DifferentiableRoom(grid, dtype=dtype, walls=WALLS, max_steps=30)
        at, _, heard = _points(shape, 40, 3)
        for q in sources:
            room.solver.add_volume_source(tuple((c + 0.5) * 0.03 for c in at[q]), np.zeros(30))
        for cell in heard:
            room.solver.add_pressure_receiver(tuple((c + 0.5) * 0.03 for c in cell))
        room.forward(30)
        return room.backward(np.random.default_rng(0).standard_normal((3, 30))).signal

    every = gradient(range(40))
    for first in range(0, 40, 20):
        np.testing.assert_array_equal(every[first:first + 20], gradient(range(first, first + 20)))
