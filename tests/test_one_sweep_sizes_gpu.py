"""From which size on runs of the two-sweep scheme take fused steps in single precision (on a GPU), from the launches
they take: two per step while the sweeps are faster, one beyond. The size in parts of L2 depends on what a step
computes and on whether its rows are ragged; the results are the same bits (test_one_sweep_runs_gpu.py)."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AbsorbingLayer, AirAbsorption, CudaAcousticFDTD, Grid, WallAdmittances

pytestmark = pytest.mark.gpu

WALLS = dict(walls=WallAdmittances(0.4, 0.1, 0.3, 0.7, 0.2, 0.05))
AIR = dict(air_absorption=AirAbsorption())
LAYER = dict(absorbing_layer=AbsorbingLayer(thickness=4))


@pytest.mark.parametrize("n, ragged, configuration, launches", [
    (156, False, WALLS, 2), (172, False, WALLS, 1), (172, True, WALLS, 2), (180, True, WALLS, 1),
    (168, False, {}, 2), (180, False, {}, 1), (168, True, {}, 2), (184, True, {}, 1),
    (136, False, {**WALLS, **AIR}, 2), (148, False, {**WALLS, **AIR}, 1),
    (144, True, {**WALLS, **AIR}, 2), (160, True, {**WALLS, **AIR}, 1),
    (144, False, AIR, 2), (156, False, AIR, 1), (160, True, AIR, 2), (184, True, AIR, 1),
    (128, False, {**WALLS, **AIR, **LAYER}, 2), (144, False, {**WALLS, **AIR, **LAYER}, 1),
    (168, True, {**WALLS, **LAYER}, 1), (168, True, LAYER, 2), (176, True, LAYER, 1),
])
def test_launches_per_step(n, ragged, configuration, launches):
    shape = (n, n + 1, n + 3) if ragged else (n, n, n)
    solver = CudaAcousticFDTD(Grid(dx=0.03, nx=shape[0], ny=shape[1], nz=shape[2]), dtype=np.float32, **configuration)
    before = solver.launch_count()
    solver.run(64)
    found = (solver.launch_count() - before) // 64
    solver.close()
    assert found == launches
