"""Forward runs recorded for the gradients (on a GPU): the recordings and the state are those of a
plain run, bit for bit, and the history they keep gives the same gradients as the two sweeps'
(which runs with checkpoints and batches of one launch per sweep use), in rooms whose rows do and do
not fill whole 16-byte chunks, for even and odd step counts, twice in a row."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AbsorbingLayer, AirAbsorption, CudaAcousticFDTD, Grid, WallAdmittances, gaussian_pulse
from ac_fdtd_b200.adjoint import DifferentiableBatch, DifferentiableRoom

pytestmark = pytest.mark.gpu

WALLS = WallAdmittances(0.2, 0.1, 0.3, 0.05, 0.4, 0.15)


def _spec(shape, layer, air):
    return dict(grid=Grid(dx=0.05, nx=shape[0], ny=shape[1], nz=shape[2]), walls=WALLS,
                absorbing_layer=AbsorbingLayer(thickness=3, faces=((1, 1), (2, 1))) if layer else None,
                air_absorption=AirAbsorption() if air else None)


def _points(spec):
    L = spec["grid"].lengths
    return [tuple(f * v for v in L) for f in (0.5, 0.02, 0.98)]


def _plain(spec, dtype, steps):
    s = CudaAcousticFDTD(spec["grid"], dtype=dtype, walls=spec["walls"], absorbing_layer=spec["absorbing_layer"],
                         air_absorption=spec["air_absorption"], steps_per_graph=0)
    points = _points(spec)
    s.add_volume_source(points[0], gaussian_pulse(steps, s.dt, 2000.0))
    for p in points[1:]:
        s.add_pressure_receiver(p)
    s.run(steps)
    return s


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape, layer, air", [
    ((13, 11, 9), True, True),       # ragged rows
    ((9, 14, 12), False, True),      # whole chunks
    ((7, 5, 1), False, False),       # a duct one cell high: both z faces in one chunk
    ((12, 10, 131), True, False),    # more chunks than one warp's row
])
@pytest.mark.parametrize("steps", [64, 71])
def test_one_room(dtype, shape, layer, air, steps):
    spec = _spec(shape, layer, air)
    wrt = ("signal", "walls", "air") if air else ("signal", "walls")
    plain = _plain(spec, dtype, steps)
    rooms = [DifferentiableRoom(spec["grid"], dtype=dtype, walls=spec["walls"],
                                absorbing_layer=spec["absorbing_layer"], air_absorption=spec["air_absorption"],
                                max_steps=80, wrt=wrt, checkpoint_every=every) for every in ((None, 16) if air else (None,))]
    gradients = []
    for room in rooms:
        points = _points(spec)
        room.solver.add_volume_source(points[0], gaussian_pulse(steps, room.dt, 2000.0))
        for p in points[1:]:
            room.solver.add_pressure_receiver(p)
        for _ in range(2):
            recorded = room.forward(steps)
            np.testing.assert_array_equal(recorded, plain.recorded_pressure)
            np.testing.assert_array_equal(room.solver.p, plain.p)
            for a, b in zip(room.solver.velocity, plain.velocity, strict=True):
                np.testing.assert_array_equal(a, b)
            gradients.append(room.backward(np.cos(np.arange(recorded.size)).reshape(recorded.shape)))
    for g in gradients[1:]:
        np.testing.assert_array_equal(g.signal, gradients[0].signal)
        np.testing.assert_array_equal(g.walls, gradients[0].walls)
        np.testing.assert_array_equal(g.initial_p, gradients[0].initial_p)
        if air:
            # the same sums over the cells, whose per-launch partials are added in the same order
            np.testing.assert_array_equal(g.strength, gradients[0].strength)
            np.testing.assert_array_equal(g.relaxation_time, gradients[0].relaxation_time)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("steps", [1, 33, 40])
def test_batch(dtype, steps):
    # rooms of a batch share their terms: every one of them has walls, a layer and air
    specs = [_spec(s, True, True) for s in ((13, 11, 9), (16, 9, 12), (8, 20, 67))]
    batch = DifferentiableBatch(specs, dtype=dtype, max_steps=40)
    for r, spec in enumerate(specs):
        points = _points(spec)
        batch.batch.add_volume_source(r, points[0], gaussian_pulse(steps, batch.batch.dt(r), 2000.0))
        for p in points[1:]:
            batch.batch.add_pressure_receiver(r, p)
    for _ in range(2):
        recorded = batch.forward(steps)
        grads = batch.backward([np.cos(np.arange(x.size)).reshape(x.shape) for x in recorded])
    for r, spec in enumerate(specs):
        plain = _plain(spec, dtype, steps)
        np.testing.assert_array_equal(recorded[r], plain.recorded_pressure)
        np.testing.assert_array_equal(batch.batch.get_field(r, 0), plain.p)
        room = DifferentiableRoom(spec["grid"], dtype=dtype, walls=spec["walls"],
                                  absorbing_layer=spec["absorbing_layer"],
                                  air_absorption=spec["air_absorption"], max_steps=40)
        points = _points(spec)
        room.solver.add_volume_source(points[0], gaussian_pulse(steps, room.dt, 2000.0))
        for p in points[1:]:
            room.solver.add_pressure_receiver(p)
        one = room.forward(steps)
        g = room.backward(np.cos(np.arange(one.size)).reshape(one.shape))
        np.testing.assert_array_equal(grads[r].signal, g.signal)
        np.testing.assert_array_equal(grads[r].walls, g.walls)
