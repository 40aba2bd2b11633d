"""Rooms with more rows than blocks of a few rows each could cover in one grid (on a GPU): 270,000 rows of 64 cells,
67,500 blocks of four rows of 32 chunks each (two doubles a chunk). Runs and recorded runs take them as the sweeps,
launched step by step, do; the gradient of a signal, in which a recording is linear, gives the recording's own
product with the weights back."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import CudaAcousticFDTD, Grid
from ac_fdtd_b200.adjoint import DifferentiableRoom

pytestmark = pytest.mark.gpu

GRID = Grid(dx=0.05, nx=1, ny=270_000, nz=64)
AT = 0.05 * 262_200.5


def _points(solver, steps):
    solver.add_volume_source((0.02, AT, 1.5), np.hanning(steps))
    solver.add_pressure_receiver((0.02, AT + 0.2, 1.4))
    solver.add_pressure_receiver((0.02, AT - 0.3, 1.7))


def test_runs():
    recorded = []
    for options in ({}, dict(steps_per_graph=0)):
        solver = CudaAcousticFDTD(GRID, dtype=np.float64, **options)
        _points(solver, 20)
        solver.run(20)
        recorded.append(solver.recorded_pressure)
        solver.close()
    assert np.any(recorded[0][:, -1])
    np.testing.assert_array_equal(*recorded)


def test_recorded_runs_and_their_gradient():
    steps = 12
    room = DifferentiableRoom(GRID, dtype=np.float64, max_steps=steps, wrt=("signal",))
    _points(room.solver, steps)
    recorded = room.forward(steps)
    weights = np.cos(np.arange(recorded.size)).reshape(recorded.shape)
    gradient = room.backward(weights)
    plain = CudaAcousticFDTD(GRID, dtype=np.float64, steps_per_graph=0)
    _points(plain, steps)
    plain.run(steps)
    np.testing.assert_array_equal(recorded, plain.recorded_pressure)
    plain.close()
    room.solver.close()
    want = float(np.sum(weights * recorded))
    # about 20 roundings per step and value, of values up to the largest recorded one
    bound = 20 * steps * np.finfo(float).eps * float(np.sum(np.abs(weights))) * float(np.max(np.abs(recorded)))
    assert abs(float(gradient.signal[0] @ np.hanning(steps)) - want) <= bound
