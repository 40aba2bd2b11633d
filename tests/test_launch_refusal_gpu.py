"""A device that refuses the cooperative launch of a room held on chip (on a GPU): the refusal is injected on the
host (``ACF_INJECT_LAUNCH_REFUSAL``). The run takes the sweeps of its scheme instead, from the step it was
refused at, and later runs do so without asking again; the results are those of any other run."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AIR, AbsorbingLayer, AirAbsorption, CudaAcousticFDTD, Grid, WallAdmittances
from oracle.leapfrog import OracleFDTD

pytestmark = pytest.mark.gpu

GRID = Grid(dx=0.02, nx=13, ny=11, nz=24)
CONFIG = dict(walls=WallAdmittances.uniform(0.2), absorbing_layer=AbsorbingLayer(thickness=3),
              air_absorption=AirAbsorption())


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("scheme", ["two_sweeps", "fused"])
def test_the_sweeps_run_instead(scheme, dtype, monkeypatch):
    oracle = OracleFDTD(GRID, AIR, dtype=dtype, **CONFIG)
    cuda = CudaAcousticFDTD(GRID, dtype=dtype, scheme=scheme, steps_per_graph=4, **CONFIG)
    for s in (oracle, cuda):
        s.p[:] = np.random.default_rng(2).standard_normal(GRID.shape).astype(dtype)
        s.add_volume_source((0.1, 0.1, 0.1), np.hanning(30))
        s.add_pressure_receiver((0.2, 0.1, 0.2))
        s.run(9)
    monkeypatch.setenv("ACF_INJECT_LAUNCH_REFUSAL", "1")
    before = cuda.launch_count()
    for s in (oracle, cuda):
        s.run(17)
    assert cuda.launch_count() - before >= 17
    monkeypatch.setenv("ACF_INJECT_LAUNCH_REFUSAL", "0")
    for s in (oracle, cuda):
        s.run(10)
    cuda.synchronize()
    np.testing.assert_array_equal(cuda.p, oracle.p)
    np.testing.assert_array_equal(cuda.recorded_pressure, oracle.recorded_pressure)
    cuda.close()
