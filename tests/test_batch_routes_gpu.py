"""Which step a batch on the fused scheme takes (on a GPU): one launch per step, but the two sweeps in single
precision where the rooms in place stay in L2 and both their copies do not. The sweeps then run in place in
whichever copy is current, so the results are those of the two-sweep scheme, bit for bit, from either copy
(timed runs take the fused step all the same, and an odd number of them changes the copy)."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AirAbsorption, Grid, RoomBatch, WallAdmittances
from ac_fdtd_b200.adjoint import DifferentiableBatch

pytestmark = pytest.mark.gpu

WALLS = WallAdmittances(0.2, 0.1, 0.3, 0.05, 0.4, 0.15)


def _specs(n, rooms, air=True):
    return [dict(grid=Grid(dx=0.03, nx=n, ny=n, nz=n), walls=WALLS,
                 air_absorption=AirAbsorption(temperature=18.0 + r) if air else None) for r in range(rooms)]


def _points(add_source, add_receiver, spec, r):
    lengths = spec["grid"].lengths
    add_source(r, tuple(0.5 * v for v in lengths), np.hanning(9))
    add_receiver(r, tuple(0.53 * v for v in lengths))


def _batch(specs, scheme, dtype=np.float32):
    batch = RoomBatch(specs, dtype=dtype, scheme=scheme, steps_per_graph=8)
    for r, spec in enumerate(specs):
        batch.set_field(r, 0, np.random.default_rng(r).standard_normal(spec["grid"].shape).astype(dtype))
        _points(batch.add_volume_source, batch.add_pressure_receiver, spec, r)
    return batch


@pytest.mark.parametrize("n, rooms, air, dtype, launches", [
    (96, 2, True, np.float32, 1),
    (108, 2, True, np.float32, 2),
    (40, 40, True, np.float32, 2),
    (124, 2, True, np.float32, 1),
    (112, 2, False, np.float32, 1),
    (120, 2, False, np.float32, 2),
    (124, 2, False, np.float32, 1),
    (92, 2, True, np.float64, 1),
])
def test_launches_per_step(n, rooms, air, dtype, launches):
    batch = RoomBatch(_specs(n, rooms, air), dtype=dtype, scheme="fused")
    before = batch.launch_count()
    batch.run(64)
    found = (batch.launch_count() - before) // 64
    batch.close()
    assert found == launches


def test_either_copy_gives_the_two_sweeps_bits():
    specs = _specs(106, 2)
    fused, swept = _batch(specs, "fused"), _batch(specs, "two_sweeps")
    for steps, timed in ((11, False), (3, True), (13, False), (9, False), (5, True), (8, False)):
        for batch in (fused, swept):
            batch.profile(timed)
            batch.run(steps)
            batch.profile(False)
        for r in range(2):
            np.testing.assert_array_equal(fused.p(r), swept.p(r))
    for r in range(2):
        for a, b in zip(fused.velocity(r), swept.velocity(r), strict=True):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(fused.recorded_pressure(r), swept.recorded_pressure(r))
    fused.close()
    swept.close()


def test_recorded_batches_take_the_same_route():
    steps = 12
    specs = _specs(106, 2)
    batch = DifferentiableBatch(specs, dtype=np.float32, max_steps=steps)
    for r, spec in enumerate(specs):
        _points(batch.batch.add_volume_source, batch.batch.add_pressure_receiver, spec, r)
    plain = RoomBatch(specs, dtype=np.float32)
    for r, spec in enumerate(specs):
        _points(plain.add_volume_source, plain.add_pressure_receiver, spec, r)
    plain.run(steps)
    before = batch.batch.launch_count()
    recorded = batch.forward(steps)
    assert (batch.batch.launch_count() - before) // steps == 2
    for r in range(2):
        np.testing.assert_array_equal(recorded[r], plain.recorded_pressure(r))
        np.testing.assert_array_equal(batch.batch.p(r), plain.p(r))
    batch.batch.close()
    plain.close()
