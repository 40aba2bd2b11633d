"""Wall maps and sums of a gradient against the numpy functions on the same boundary sums (on a GPU):
the maps bit for bit; the sums, of at most 2100 doubles in two orders, to 4200 half-ulps of the sum
of magnitudes."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import Grid, WallAdmittances, _native, gaussian_pulse
from ac_fdtd_b200.adjoint import DifferentiableBatch, DifferentiableRoom, wall_gradients
from ac_fdtd_b200.boundaries import WallPatches
from ac_fdtd_b200.solver import _as_double_pointer

pytestmark = pytest.mark.gpu

STEPS = 40


def _close(found, walls, shape, shell, block, c):
    sums, cells = wall_gradients(walls, shape, shell, c, block.dt, block.dx)
    for a, b in zip(found.wall_cells, cells, strict=True):
        np.testing.assert_array_equal(a, b)
    bound = 4200 * 2.0**-53 * sum(np.abs(m).sum() for m in cells)
    assert found.walls.shape == sums.shape
    np.testing.assert_allclose(found.walls, sums, rtol=0.0, atol=bound)


def _walls(patches, seed):
    if patches == 0:
        return WallAdmittances(0.2, 0.1, 0.3, 0.05, 0.4, 0.15)
    return WallPatches(np.random.default_rng(seed).uniform(0.05, 0.6, (6, patches, patches)))


@pytest.mark.parametrize("shape", [(13, 11, 9), (1, 6, 5), (7, 1, 33), (52, 40, 1), (50, 34, 41)])
@pytest.mark.parametrize("patches", [0, 1, 3, 12])      # 12: more patches than cells along some axes
def test_one_room(shape, patches):
    walls = _walls(patches, 3)
    grid = Grid(dx=0.05, nx=shape[0], ny=shape[1], nz=shape[2])
    room = DifferentiableRoom(grid, dtype=np.float64, walls=walls, max_steps=STEPS)
    s = room.solver
    s.add_volume_source(tuple(0.4 * v for v in grid.lengths), gaussian_pulse(STEPS, room.dt, 2000.0))
    s.add_pressure_receiver(tuple(0.7 * v for v in grid.lengths))
    recorded = room.forward(STEPS)
    found = room.backward(recorded)
    shell = np.zeros(s._lib.acf_adjoint_shell_size(s._handle))
    grad = np.ascontiguousarray(recorded, dtype=np.float64)
    _native.check(s._lib.acf_adjoint_run(s._handle, _as_double_pointer(grad), None, _as_double_pointer(shell), None,
                                         s._stream), "acf_adjoint_run")
    _close(found, walls, shape, shell, s.coefficients, float(s.medium.sound_speed))


def test_rooms_of_a_batch():
    shapes = [(13, 11, 9), (20, 16, 25)]
    specs = [dict(grid=Grid(dx=0.05, nx=s[0], ny=s[1], nz=s[2]), walls=_walls(p, r))
             for r, (s, p) in enumerate(zip(shapes, (0, 4)))]
    batch = DifferentiableBatch(specs, dtype=np.float64, max_steps=STEPS)
    b = batch.batch
    for r, spec in enumerate(specs):
        b.add_volume_source(r, tuple(0.4 * v for v in spec["grid"].lengths), gaussian_pulse(STEPS, b.dt(r), 2000.0))
        b.add_pressure_receiver(r, tuple(0.7 * v for v in spec["grid"].lengths))
    recorded = batch.forward(STEPS)
    found = batch.backward(recorded)
    sizes = [b._lib.acf_batch_adjoint_shell_size(b._handle, r) for r in range(2)]
    shell = np.zeros(sum(sizes))
    grad = np.ascontiguousarray(np.concatenate(recorded), dtype=np.float64)
    _native.check(b._lib.acf_batch_adjoint_run(b._handle, _as_double_pointer(grad), None, _as_double_pointer(shell),
                                               b._stream), "acf_batch_adjoint_run")
    from ac_fdtd_b200.medium import AIR
    for r, part in enumerate(np.split(shell, [sizes[0]])):
        _close(found[r], specs[r]["walls"], shapes[r], part, b.blocks[r], float(AIR.sound_speed))


def test_refused_without_a_run_or_outputs():
    grid = Grid(dx=0.05, nx=6, ny=5, nz=4)
    room = DifferentiableRoom(grid, dtype=np.float64, max_steps=STEPS)
    s = room.solver
    out = np.zeros(1000)
    call = s._lib.acf_adjoint_wall_gradients
    assert call(s._handle, 1.0, 1, _as_double_pointer(out), _as_double_pointer(out), s._stream) != 0    # no run
    room.forward(8)
    assert call(s._handle, 1.0, 0, _as_double_pointer(out), _as_double_pointer(out), s._stream) != 0
    assert call(s._handle, 1.0, 1, None, _as_double_pointer(out), s._stream) != 0
