"""Which step a recorded run of a batch takes (on a GPU), from its launches: one fused step per step, or the two sweeps
in place where those are faster, which is another range of sizes than for plain runs. Recordings, state and gradients
are the same bits on both sides: each room alone is the reference."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AbsorbingLayer, AirAbsorption, CudaAcousticFDTD, Grid, RoomBatch, WallAdmittances
from ac_fdtd_b200.adjoint import DifferentiableBatch

pytestmark = pytest.mark.gpu

STEPS = 12


def _specs(n, rooms, air, layer):
    return [dict(grid=Grid(dx=0.03, nx=n, ny=n, nz=n), walls=WallAdmittances(0.2, 0.1, 0.3, 0.05, 0.4, 0.15),
                 absorbing_layer=AbsorbingLayer(thickness=4) if layer else None,
                 air_absorption=AirAbsorption(temperature=18.0 + r) if air else None) for r in range(rooms)]


@pytest.mark.parametrize("n, rooms, air, layer, dtype, launches", [
    (100, 2, False, False, np.float32, 1), (112, 2, False, False, np.float32, 2), (128, 2, False, False, np.float32, 1),
    (104, 2, False, True, np.float32, 1), (116, 2, False, True, np.float32, 2), (128, 2, False, True, np.float32, 1),
    (100, 2, True, False, np.float32, 1), (108, 2, True, False, np.float32, 2), (124, 2, True, False, np.float32, 1),
    (108, 2, True, True, np.float32, 1),
    (88, 2, False, False, np.float64, 1), (96, 2, False, False, np.float64, 2), (104, 2, False, False, np.float64, 1),
    (96, 2, True, False, np.float64, 1),
])
def test_route_and_results(n, rooms, air, layer, dtype, launches):
    specs = _specs(n, rooms, air, layer)
    batch = DifferentiableBatch(specs, dtype=dtype, max_steps=STEPS)
    alone = []
    for r, spec in enumerate(specs):
        lengths = spec["grid"].lengths
        solver = CudaAcousticFDTD(dtype=dtype, steps_per_graph=0, **spec)
        for add_source, add_receiver in ((lambda *a: batch.batch.add_volume_source(r, *a),
                                          lambda p: batch.batch.add_pressure_receiver(r, p)),
                                         (solver.add_volume_source, solver.add_pressure_receiver)):
            add_source(tuple(0.5 * v for v in lengths), np.hanning(9))
            add_receiver(tuple(0.53 * v for v in lengths))
        solver.run(STEPS)
        alone.append(solver)
    before = batch.batch.launch_count()
    recorded = batch.forward(STEPS)
    found = (batch.batch.launch_count() - before) // STEPS
    for r, solver in enumerate(alone):
        np.testing.assert_array_equal(recorded[r], solver.recorded_pressure)
        np.testing.assert_array_equal(batch.batch.p(r), solver.p)
        solver.close()
    batch.batch.close()
    assert found == launches


@pytest.mark.parametrize("layer, launches", [(False, 2), (True, 1)])
def test_plain_batches_with_a_layer_take_the_fused_step(layer, launches):
    """A layer costs the sweeps more than the fused step: without relaxation states only rooms without one take them."""
    batch = RoomBatch(_specs(118, 2, False, layer), dtype=np.float32, scheme="fused")
    before = batch.launch_count()
    batch.run(64)
    found = (batch.launch_count() - before) // 64
    batch.close()
    assert found == launches
