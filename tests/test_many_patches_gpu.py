"""Wall gradients of walls with more patches than the device sums (on a GPU): as with any other number of patches,
each patch gets the sum of its cells, and patches without a cell get nothing."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import Grid
from ac_fdtd_b200.adjoint import DifferentiableRoom
from ac_fdtd_b200.boundaries import FACES, WallPatches, patch_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("patches", [1024, 1025, 1300])
def test_patches_are_the_sums_of_their_cells(patches):
    shape = (9, 12, 7)
    room = DifferentiableRoom(Grid(dx=0.05, nx=shape[0], ny=shape[1], nz=shape[2]), dtype=np.float64, max_steps=20,
                              walls=WallPatches(np.full((6, patches, patches), 0.2)), wrt=("signal", "walls"))
    room.solver.add_volume_source((0.2, 0.2, 0.2), np.hanning(9))
    room.solver.add_pressure_receiver((0.3, 0.4, 0.2))
    recorded = room.forward(20)
    gradients = room.backward(np.cos(np.arange(recorded.size)).reshape(recorded.shape))
    assert gradients.walls.shape == (6, patches, patches)
    for f, (axis, _) in enumerate(FACES):
        b, c = [a for a in range(3) if a != axis]
        at = np.ix_(patch_index(shape[b], patches), patch_index(shape[c], patches))   # a cell per patch at most
        assert np.any(gradients.wall_cells[f])
        np.testing.assert_array_equal(gradients.walls[f][at], gradients.wall_cells[f])
        assert np.count_nonzero(gradients.walls[f]) == np.count_nonzero(gradients.wall_cells[f])
    room.solver.close()
