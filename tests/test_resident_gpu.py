"""Rooms held on chip: many steps per launch (``csrc/acfdtd_resident_kernel.cuh``) on a GPU.

A single room on the two-sweep or fused scheme whose state fits the GPU takes runs of eight steps or
more in one cooperative launch. Its pin is the sweeps it replaces, launched step by step
(``steps_per_graph=0``), and the oracle: every field, relaxation state and recording bit for bit.
The shapes reach one to eight x planes per thread, bricks cut short at either end, one-cell axes, rows
that end inside a chunk, a row of one chunk and one CTA; the runs reach the split of long runs.
"""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import (
    AIR,
    AbsorbingLayer,
    AirAbsorption,
    CudaAcousticFDTD,
    Grid,
    WallAdmittances,
)
from ac_fdtd_b200._native import ERR_STATE, NativeError
from ac_fdtd_b200.adjoint import FixedProcesses
from oracle.leapfrog import OracleFDTD

pytestmark = pytest.mark.gpu

EVERYTHING = dict(walls=WallAdmittances(0.4, 0.1, 0.0, 0.7, 0.2, 0.05),
                  absorbing_layer=AbsorbingLayer(thickness=3), air_absorption=AirAbsorption())
SMALL = [(1, 1, 1), (1, 1, 4), (2, 9, 5), (6, 1, 8), (5, 7, 300), (13, 11, 24), (20, 17, 15), (33, 70, 9)]


def _filled(solver, shape, dtype):
    dx = solver.grid.dx
    last = tuple((n - 0.5) * dx for n in shape)
    solver.p[:] = np.random.default_rng(1).standard_normal(shape).astype(dtype)
    solver.add_volume_source((0.0, 0.0, 0.0), np.hanning(30))
    solver.add_volume_source(last, np.hanning(9))
    solver.add_volume_source(last, np.hanning(12))
    solver.add_pressure_receiver(last)
    solver.add_pressure_receiver(tuple(0.5 * v for v in last))
    return solver


def _same(a, b):
    np.testing.assert_array_equal(a.p, b.p)
    for x, y in zip(a.velocity, b.velocity, strict=True):
        np.testing.assert_array_equal(x, y)
    for x, y in zip(a.relaxation_states, b.relaxation_states, strict=True):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(a.recorded_pressure, b.recorded_pressure)


def _pair(shape, dtype, configuration, scheme="two_sweeps"):
    grid = Grid(dx=0.02, nx=shape[0], ny=shape[1], nz=shape[2])
    held = CudaAcousticFDTD(grid, dtype=dtype, scheme=scheme, **configuration)
    swept = CudaAcousticFDTD(grid, dtype=dtype, scheme=scheme, steps_per_graph=0, **configuration)
    return grid, _filled(held, shape, dtype), _filled(swept, shape, dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", SMALL)
def test_resident_steps_equal_the_sweeps_and_the_oracle(shape, dtype):
    grid, held, swept = _pair(shape, dtype, EVERYTHING)
    oracle = OracleFDTD(grid, AIR, dtype=dtype, **EVERYTHING)
    _filled(oracle, shape, dtype)
    launches = held.launch_count()
    for n in (9, 16, 8):
        for s in (held, swept, oracle):
            s.run(n)
    assert held.launch_count() - launches <= 8          # not a launch per step
    held.synchronize()
    _same(held, swept)
    np.testing.assert_array_equal(held.p, oracle.p)
    np.testing.assert_array_equal(held.recorded_pressure, oracle.recorded_pressure)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", [(64, 64, 64), (80, 77, 83), (97, 91, 77), (101, 110, 99), (128, 122, 127)])
def test_larger_rooms_equal_the_sweeps(shape, dtype):
    """Two to eight planes per thread (and, in double precision, rooms that are too large)."""
    for configuration in ({"walls": WallAdmittances.uniform(0.3)}, EVERYTHING):
        _, held, swept = _pair(shape, dtype, configuration, scheme="fused")
        for s in (held, swept):
            s.run(11)
            s.run(8)
        held.synchronize()
        _same(held, swept)
        held.close()
        swept.close()


@pytest.mark.parametrize("air", [AirAbsorption(relaxation=False), AirAbsorption(classical=False),
                                 FixedProcesses([1e-3, 2e-3, 5e-4, 1e-4], [1e-4, 2e-5, 3e-4, 6e-5])])
def test_one_two_and_four_relaxation_states(air):
    for shape in ((21, 18, 22), (90, 90, 90)):
        _, held, swept = _pair(shape, np.float32, dict(air_absorption=air))
        for s in (held, swept):
            s.run(20)
        _same(held, swept)
        held.close()
        swept.close()


@pytest.mark.parametrize("steps", [2048, 2049, 2050])
def test_runs_longer_than_one_launch(steps):
    _, held, swept = _pair((9, 8, 10), np.float32, EVERYTHING)
    for s in (held, swept):
        s.run(steps)
    _same(held, swept)


def test_waits_are_bounded():
    """The first CTA stops sending at step 5: its neighbours' 5 ms waits run out, the run reports
    it, and after a reset the same handle is right again."""
    shape = (24, 20, 16)
    _, held, swept = _pair(shape, np.float32, EVERYTHING)
    from ac_fdtd_b200 import _native

    _native.check(held._lib.acf_set_wait_test(held._handle, 5_000_000, 5), "acf_set_wait_test")
    held.run(20)
    with pytest.raises(NativeError) as error:
        held.synchronize()
    assert error.value.status == ERR_STATE
    _native.check(held._lib.acf_set_wait_test(held._handle, 0, -1), "acf_set_wait_test")
    held.reset_state()
    swept.reset_state()
    held.step_index = swept.step_index = 0
    for s in (held, swept):
        s.run(30)
    held.synchronize()
    _same(held, swept)
