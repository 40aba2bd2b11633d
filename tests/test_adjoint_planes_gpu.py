"""The adjoint chunk step takes fewer planes per block where a room would leave SMs idle (on a GPU): gradients of a
cell do not depend on it, bit for bit, and the air sums, added in another grouping, agree to their rounding: some 1e5
terms in double precision, 1e5 x 1.1e-16 of their largest partial sum, 1e-9 of a total that cancels a hundredfold."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AirAbsorption, Grid, WallAdmittances
from ac_fdtd_b200.adjoint import DifferentiableRoom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(20, 21, 23), (3, 40, 9), (60, 61, 63)])     # a few, a few tens, hundreds of blocks
def test_planes_per_block_leave_gradients_alone(shape):
    steps, out = 30, []
    for planes in (4, 1, 3, 16):
        room = DifferentiableRoom(Grid(dx=0.05, nx=shape[0], ny=shape[1], nz=shape[2]), dtype=np.float64,
                                  walls=WallAdmittances(0.2, 0.1, 0.3, 0.05, 0.4, 0.15), air_absorption=AirAbsorption(),
                                  max_steps=steps, wrt=("signal", "walls", "air"))
        room.solver.set_launch(128, planes)
        lengths = room.solver.grid.lengths
        room.solver.add_volume_source(tuple(0.5 * v for v in lengths), np.hanning(9))
        room.solver.add_pressure_receiver(tuple(0.6 * v for v in lengths))
        recorded = room.forward(steps)
        out.append(room.backward(np.cos(np.arange(recorded.size)).reshape(recorded.shape)))
        room.solver.close()
    for other in out[1:]:
        for name in ("signal", "walls", "initial_p"):
            np.testing.assert_array_equal(getattr(out[0], name), getattr(other, name))
        for name in ("strength", "relaxation_time"):
            a, b = getattr(out[0], name), getattr(other, name)
            assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(a)), name
