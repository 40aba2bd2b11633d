"""The steps that runs of small rooms no longer reach by default, since those rooms are held on chip (on a GPU):
the two sweeps and the lean and the chunk step, launched step by step and replayed from graphs (runs of
fewer than eight steps take those), on small and degenerate rooms, with and without the L2 prefetch and for
each number of planes per block. Against the oracle: every field, relaxation state and recording bit for bit,
and the launches show that they ran."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import AIR, AbsorbingLayer, AirAbsorption, CudaAcousticFDTD, Grid, WallAdmittances
from oracle.leapfrog import OracleFDTD

pytestmark = pytest.mark.gpu

SHAPES = [(13, 11, 24), (1, 1, 4), (6, 1, 8), (2, 9, 4), (9, 10, 40), (5, 3, 12), (4, 37, 132), (13, 11, 23),
          (6, 1, 5), (2, 9, 1), (1, 1, 2), (5, 3, 7), (4, 37, 133), (7, 6, 6)]
FACES = [None, ((0, 0), (0, 1)), ((1, 1), (2, 0))]


def _configuration(faces):
    layer = AbsorbingLayer(thickness=3) if faces is None else AbsorbingLayer(thickness=3, faces=faces)
    return dict(walls=WallAdmittances(0.4, 0.1, 0.0, 0.7, 0.2, 0.05), absorbing_layer=layer,
                air_absorption=AirAbsorption())


def _prepared(solver, shape, dtype):
    corner = tuple((n - 0.5) * 0.02 for n in shape)
    solver.p[:] = np.random.default_rng(sum(shape)).standard_normal(shape).astype(dtype)
    solver.add_volume_source((0.0, 0.0, 0.0), np.hanning(12))
    solver.add_volume_source(corner, np.hanning(7))
    solver.add_pressure_receiver(corner)
    solver.add_pressure_receiver((0.0, corner[1], 0.0))
    return solver


def _same(cuda, oracle):
    np.testing.assert_array_equal(cuda.p, oracle.p)
    for axis in range(3):
        np.testing.assert_array_equal(cuda.velocity[axis], oracle.velocity[axis])
    np.testing.assert_array_equal(cuda.recorded_pressure, oracle.recorded_pressure)
    for got, (want, *_rest) in zip(cuda.relaxation_states, oracle.relax, strict=True):
        np.testing.assert_array_equal(got, want)


def _oracle(shape, dtype, configuration, steps):
    grid = Grid(dx=0.02, nx=shape[0], ny=shape[1], nz=shape[2])
    oracle = _prepared(OracleFDTD(grid, AIR, dtype=dtype, **configuration), shape, dtype)
    oracle.run(steps)
    return grid, oracle


@pytest.mark.parametrize("scheme", ["two_sweeps", "fused"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("faces", FACES)
def test_steps_and_graph_replays_match_the_oracle(faces, dtype, scheme):
    configuration = _configuration(faces)
    per_step = 2 if scheme == "two_sweeps" else 1
    for shape in SHAPES:
        grid, oracle = _oracle(shape, dtype, configuration, 33)
        for steps_per_graph, runs in ((0, (33,)), (3, (7, 6, 7, 6, 7)), (2, (7, 5, 7, 7, 7))):
            for prefetch in (False, True):
                cuda = CudaAcousticFDTD(grid, dtype=dtype, scheme=scheme, steps_per_graph=steps_per_graph,
                                        **configuration)
                cuda.set_prefetch(prefetch)
                _prepared(cuda, shape, dtype)
                before = cuda.launch_count()
                for n in runs:
                    cuda.run(n)
                assert cuda.launch_count() - before >= 33 * per_step
                _same(cuda, oracle)
                cuda.close()


@pytest.mark.parametrize("scheme", ["two_sweeps", "fused"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("planes", [1, 3, 16])
def test_plane_groups_match_the_oracle(planes, dtype, scheme):
    shape = (26, 12, 37)
    configuration = _configuration(((0, 0), (0, 1)))
    grid, oracle = _oracle(shape, dtype, configuration, 21)
    for steps_per_graph in (0, 2, 4):
        cuda = CudaAcousticFDTD(grid, dtype=dtype, scheme=scheme, steps_per_graph=steps_per_graph, **configuration)
        cuda.set_launch(64, planes)
        _prepared(cuda, shape, dtype)
        before = cuda.launch_count()
        for _ in range(3):
            cuda.run(7)
        assert cuda.launch_count() - before >= 21
        _same(cuda, oracle)
        cuda.close()


def test_switching_schemes_between_steps():
    shape = (13, 11, 23)
    configuration = _configuration(None)
    grid, oracle = _oracle(shape, np.float32, configuration, 36)
    cuda = _prepared(CudaAcousticFDTD(grid, dtype=np.float32, steps_per_graph=4, **configuration), shape, np.float32)
    for scheme, n in (("two_sweeps", 7), ("fused", 5), ("staged", 3), ("fused", 16), ("two_sweeps", 5)):
        cuda.set_scheme(scheme)      # sixteen steps of the fused scheme are held on chip, from the copy that is current
        cuda.run(n)
    _same(cuda, oracle)
    cuda.close()
