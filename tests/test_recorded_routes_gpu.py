"""Which step a recorded forward run takes, and that it does not show in the results (on a GPU): one
launch per step where both copies of the room and the history go well with L2, the two sweeps in place
where only the room in place does; the history of either gives the same gradients, bit for bit, as
runs with checkpoints, which always take the sweeps."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AirAbsorption, Grid, WallAdmittances, gaussian_pulse
from ac_fdtd_b200.adjoint import DifferentiableRoom

pytestmark = pytest.mark.gpu

STEPS = 12


def _run(shape, dtype, every):
    grid = Grid(dx=0.03, nx=shape[0], ny=shape[1], nz=shape[2])
    room = DifferentiableRoom(grid, dtype=dtype, walls=WallAdmittances(0.2, 0.1, 0.3, 0.05, 0.4, 0.15),
                              air_absorption=AirAbsorption(), max_steps=STEPS, wrt=("signal", "walls", "air"),
                              checkpoint_every=every)
    s = room.solver
    s.add_volume_source(tuple(0.5 * v for v in grid.lengths), gaussian_pulse(STEPS, room.dt, 3000.0))
    s.add_pressure_receiver(tuple(0.53 * v for v in grid.lengths))
    before = s.launch_count()
    recorded = room.forward(STEPS)
    launches = (s.launch_count() - before) // STEPS
    g = room.backward(np.cos(np.arange(STEPS))[None])
    out = [recorded, s.p.copy(), g.signal, g.walls, g.initial_p, g.strength, g.relaxation_time]
    s.close()
    return launches, out


@pytest.mark.parametrize("shape, dtype, launches", [
    ((96, 96, 96), np.float32, 1),       # both copies in L2 beside the history
    ((128, 128, 128), np.float32, 2),    # in place only
    ((164, 168, 172), np.float32, 1),    # neither
    ((97, 131, 77), np.float32, 2),      # ragged rows
    ((60, 61, 63), np.float32, 1),
    ((88, 88, 88), np.float64, 1),
    ((96, 96, 96), np.float64, 2),
    ((104, 104, 104), np.float64, 1),
])
def test_route_and_results(shape, dtype, launches):
    found, out = _run(shape, dtype, None)
    assert found == launches
    swept, want = _run(shape, dtype, 5)
    assert swept == 2
    for a, b in zip(out, want, strict=True):
        np.testing.assert_array_equal(a, b)
