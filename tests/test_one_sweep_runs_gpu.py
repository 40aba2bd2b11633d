"""Long runs on the two-sweep scheme that take fused steps inside (on a GPU): the same bits as the sweeps
launched step by step, for even and odd step counts, with the state in the room's own copy after each
run, through graphs, state access between runs, and a switch of scheme."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AbsorbingLayer, AirAbsorption, CudaAcousticFDTD, Grid, WallAdmittances

pytestmark = pytest.mark.gpu

EVERYTHING = dict(walls=WallAdmittances(0.4, 0.1, 0.0, 0.7, 0.2, 0.05),
                  absorbing_layer=AbsorbingLayer(thickness=3), air_absorption=AirAbsorption())


def _solver(shape, dtype, configuration, **options):
    dx = 0.02
    s = CudaAcousticFDTD(Grid(dx=dx, nx=shape[0], ny=shape[1], nz=shape[2]), dtype=dtype, **configuration, **options)
    s.p[:] = np.random.default_rng(1).standard_normal(shape).astype(dtype)
    last = tuple((n - 0.5) * dx for n in shape)
    s.add_volume_source((0.0, 0.0, 0.0), np.hanning(60))
    s.add_volume_source(last, np.hanning(9))
    s.add_pressure_receiver(last)
    s.add_pressure_receiver(tuple(0.5 * v for v in last))
    return s


@pytest.mark.parametrize("dtype, shape, configuration", [
    (np.float64, (112, 111, 113), {"walls": WallAdmittances.uniform(0.3)}),
    (np.float64, (111, 114, 112), EVERYTHING),
    (np.float32, (150, 141, 143), EVERYTHING),
    (np.float32, (177, 176, 180), {}),
])
def test_runs_equal_the_sweeps(dtype, shape, configuration):
    fast = _solver(shape, dtype, configuration)
    slow = _solver(shape, dtype, configuration, steps_per_graph=0)
    pointer = fast.field_pointer(0)
    for n in (8, 9, 70, 3, 67):
        before = fast.launch_count()
        fast.run(n)
        slow.run(n)
        if n >= 8:
            assert fast.launch_count() - before < 2 * n      # not two launches a step
        assert fast.field_pointer(0) == pointer              # the caller's copy
    np.testing.assert_array_equal(fast.p, slow.p)
    fast.p[1:4] *= 0.5
    slow.p[1:4] *= 0.5
    fast.set_scheme("fused")
    slow.set_scheme("fused")
    fast.run(5)
    slow.run(5)
    fast.set_scheme("two_sweeps")
    slow.set_scheme("two_sweeps")
    fast.run(12)
    slow.run(12)
    fast.synchronize()
    np.testing.assert_array_equal(fast.p, slow.p)
    for a, b in zip(fast.velocity, slow.velocity, strict=True):
        np.testing.assert_array_equal(a, b)
    for a, b in zip(fast.relaxation_states, slow.relaxation_states, strict=True):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(fast.recorded_pressure, slow.recorded_pressure)
    fast.close()
    slow.close()
