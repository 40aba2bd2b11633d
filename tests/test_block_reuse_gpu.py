"""Device memory that handles give back is kept for the next ones (on a GPU): what a solver computes
does not depend on who used its memory before, what is kept is bounded, and solvers made and closed by
several threads at once do not meet in it."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from ac_fdtd_b200 import AIR, AirAbsorption, CudaAcousticFDTD, Grid, RoomBatch, WallAdmittances
from oracle.leapfrog import OracleFDTD

pytestmark = pytest.mark.gpu

CONFIG = dict(walls=WallAdmittances(0.4, 0.1, 0.0, 0.7, 0.2, 0.05), air_absorption=AirAbsorption())


def _run(make, shape, seed, scheme):
    grid = Grid(dx=0.03, nx=shape[0], ny=shape[1], nz=shape[2])
    solver = make(grid, scheme)
    solver.p[:] = np.random.default_rng(seed).standard_normal(shape).astype(np.float32)
    solver.add_volume_source((0.1, 0.1, 0.1), np.hanning(12))
    solver.add_pressure_receiver((0.2, 0.2, 0.2))
    solver.run(13)
    out = np.array(solver.p), solver.recorded_pressure
    if hasattr(solver, "close"):
        solver.close()
    return out


def _cuda(grid, scheme):
    return CudaAcousticFDTD(grid, dtype=np.float32, scheme=scheme, **CONFIG)


def _oracle(grid, scheme):
    return OracleFDTD(grid, AIR, dtype=np.float32, **CONFIG)


def test_a_new_solver_on_used_memory_is_like_any_other():
    shapes = [(20, 17, 15), (19, 17, 15), (24, 20, 30), (20, 17, 15), (9, 31, 18)]
    for n, shape in enumerate(shapes * 3):
        scheme = ("two_sweeps", "fused", "staged")[n % 3]
        got, want = _run(_cuda, shape, n, scheme), _run(_oracle, shape, n, scheme)
        for a, b in zip(got, want, strict=True):
            np.testing.assert_array_equal(a, b)


def test_what_is_kept_is_bounded():
    torch = pytest.importorskip("torch")
    solver = CudaAcousticFDTD(Grid(dx=0.03, nx=40, ny=40, nz=40), dtype=np.float32)
    solver.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for n in range(12):             # 150 MB of different sizes each
        grid = Grid(dx=0.03, nx=140 + 2 * n, ny=150, nz=200)
        RoomBatch([dict(grid=grid), dict(grid=Grid(dx=0.03, nx=30 + n, ny=20, nz=24))]).close()
    assert before - torch.cuda.mem_get_info()[0] <= 300 << 20


def test_threads_make_and_close_solvers_at_once():
    wanted = {shape: _run(_oracle, shape, 3, "two_sweeps") for shape in ((20, 17, 15), (24, 20, 30))}
    wrong = []

    def work(shape):
        for _ in range(8):
            got = _run(_cuda, shape, 3, "two_sweeps")
            if not all(np.array_equal(a, b) for a, b in zip(got, wanted[shape])):
                wrong.append(shape)

    threads = [threading.Thread(target=work, args=(shape,)) for shape in list(wanted) * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
