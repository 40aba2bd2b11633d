"""Which rooms a run holds on chip (on a GPU), from the launches it takes: those where that is faster than
the step of the scheme they are on, in two launches per run; the others take a launch or two per step. (All
give the same bits, which test_resident_gpu.py and test_parity_gpu.py hold.)"""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AbsorbingLayer, AirAbsorption, CudaAcousticFDTD, Grid, WallAdmittances

pytestmark = pytest.mark.gpu

WALLS = dict(walls=WallAdmittances(0.4, 0.1, 0.3, 0.7, 0.2, 0.05))
AIR = dict(WALLS, air_absorption=AirAbsorption())
ALL = dict(AIR, absorbing_layer=AbsorbingLayer(thickness=4))


@pytest.mark.parametrize("scheme, dtype, n, configuration, held", [
    ("fused", np.float32, 96, ALL, True),
    ("fused", np.float32, 100, AIR, True),
    ("fused", np.float32, 100, ALL, False),
    ("fused", np.float32, 108, WALLS, True),
    ("fused", np.float32, 108, AIR, False),
    ("fused", np.float32, 108, ALL, False),
    ("fused", np.float32, 128, WALLS, False),
    ("two_sweeps", np.float32, 108, ALL, True),
    ("two_sweeps", np.float32, 128, WALLS, True),
    ("two_sweeps", np.float64, 72, ALL, True),
    ("two_sweeps", np.float64, 80, ALL, False),
    ("two_sweeps", np.float64, 88, AIR, True),
    ("fused", np.float64, 96, WALLS, False),
])
def test_rooms_are_held_where_that_is_faster(scheme, dtype, n, configuration, held):
    steps = 64
    solver = CudaAcousticFDTD(Grid(dx=0.03, nx=n, ny=n, nz=n), dtype=dtype, scheme=scheme, **configuration)
    before = solver.launch_count()
    solver.run(steps)
    launches = solver.launch_count() - before
    solver.synchronize()
    solver.close()
    assert launches == 2 if held else launches >= steps
