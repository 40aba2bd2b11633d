"""Tuning a small room on a GPU leaves its runs held on chip, two launches for any number of steps."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import CudaAcousticFDTD, Grid, WallAdmittances
from ac_fdtd_b200.autotune import apply_tuned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_a_tuned_small_room_stays_held(dtype):
    solver = CudaAcousticFDTD(Grid(dx=0.03, nx=47, ny=44, nz=51), dtype=dtype, walls=WallAdmittances.uniform(0.3))
    chosen = apply_tuned(solver)
    before = solver.launch_count()
    solver.run(64)
    assert solver.launch_count() - before == 2, chosen
    solver.close()
