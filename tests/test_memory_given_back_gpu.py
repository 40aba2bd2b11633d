"""Device memory that the library could do without (on a GPU): blocks kept for the next handle are bounded and
given back on request, and a second copy of p and v that a run on the two-sweep scheme allocated gives way to an
allocation that would fail otherwise, or to a request; the runs after that have the same results."""

from __future__ import annotations

import gc
import threading

import numpy as np
import pytest

import ac_fdtd_b200
from ac_fdtd_b200 import AirAbsorption, CudaAcousticFDTD, Grid, RoomBatch, WallAdmittances
from ac_fdtd_b200.adjoint import DifferentiableBatch

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _grid(nx, ny, nz):
    return Grid(dx=0.03, nx=nx, ny=ny, nz=nz)


def _free(torch):
    gc.collect()                     # solvers that other tests left to the collector
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _solver(n, dtype=np.float64, **options):
    solver = CudaAcousticFDTD(_grid(n, n, n), dtype=dtype, walls=WallAdmittances.uniform(0.3), **options)
    solver.add_volume_source((0.1, 0.1, 0.1), np.hanning(40))
    solver.add_pressure_receiver((0.3, 0.2, 0.2))
    return solver


def test_idle_blocks_are_bounded_and_given_back():
    """Twelve batches, open together, of two rooms whose state is one block of 24 to 46 MB: each small enough to be
    kept, 420 MB in all."""
    torch = pytest.importorskip("torch")
    CudaAcousticFDTD(_grid(40, 40, 40), dtype=np.float32).close()
    ac_fdtd_b200.release_memory()
    before = _free(torch)
    batches = [RoomBatch([dict(grid=_grid(60 + 5 * n, 100, 200)), dict(grid=_grid(8, 9, 10))]) for n in range(12)]
    assert before - _free(torch) > 350 * MB
    for batch in batches:
        batch.close()
    kept = before - _free(torch)
    assert 100 * MB < kept <= 256 * MB + 16 * MB       # the bound, and what the driver rounds up
    ac_fdtd_b200.release_memory()
    assert before - _free(torch) <= 16 * MB


def test_a_second_copy_gives_way_to_an_allocation():
    torch = pytest.importorskip("torch")
    first, plain = _solver(320), _solver(320, steps_per_graph=0)
    before = _free(torch)
    first.run(10)                                  # takes fused steps, and a second copy of 1.1 GB
    assert before - _free(torch) > 1000 * MB
    filler = torch.empty(_free(torch) - 600 * MB, dtype=torch.uint8, device="cuda")
    try:
        second = _solver(300)                      # 0.9 GB
    finally:
        del filler
        torch.cuda.empty_cache()
    for n in (9, 12):
        first.run(n)
    plain.run(31)
    np.testing.assert_array_equal(first.p, plain.p)
    np.testing.assert_array_equal(first.recorded_pressure, plain.recorded_pressure)
    for s in (first, second, plain):
        s.close()


def test_second_copies_are_given_back_on_request():
    """Between the runs of a single room, and between the two halves of a batch's gradient."""
    torch = pytest.importorskip("torch")
    solver, plain = _solver(150), _solver(150, steps_per_graph=0)
    specs = [dict(grid=_grid(24, 20, 30), walls=WallAdmittances.uniform(0.2), air_absorption=AirAbsorption())
             for _ in range(2)]
    gradients = []
    for released in (False, True):
        batch = DifferentiableBatch(specs, dtype=np.float32, max_steps=20)
        for r in range(2):
            batch.batch.add_volume_source(r, (0.2, 0.2, 0.2), np.hanning(9))
            batch.batch.add_pressure_receiver(r, (0.4, 0.3, 0.5))
        for _ in range(2):
            recorded = batch.forward(20)
            if released:
                ac_fdtd_b200.release_memory()
            gradients.append(batch.backward([np.cos(np.arange(x.size)).reshape(x.shape) for x in recorded]))
        batch.batch.close()
    for other in gradients[1:]:
        for a, b in zip(gradients[0], other, strict=True):
            np.testing.assert_array_equal(a.signal, b.signal)
            np.testing.assert_array_equal(a.walls, b.walls)
    for n in (10, 11, 3, 16):
        solver.run(n)
        held = _free(torch)
        ac_fdtd_b200.release_memory()
        if n >= 8:
            assert _free(torch) - held > 100 * MB
    plain.run(40)
    np.testing.assert_array_equal(solver.p, plain.p)
    np.testing.assert_array_equal(solver.recorded_pressure, plain.recorded_pressure)
    solver.close()
    plain.close()


def test_released_by_one_thread_while_others_run():
    plain = _solver(150, np.float64, steps_per_graph=0)
    plain.run(80)
    want = np.array(plain.p)
    plain.close()
    stop, wrong = threading.Event(), []

    def work():
        solver = _solver(150)
        for _ in range(8):
            solver.run(10)
        if not np.array_equal(solver.p, want):
            wrong.append(1)
        solver.close()

    def release():
        while not stop.is_set():
            ac_fdtd_b200.release_memory()

    workers = [threading.Thread(target=work) for _ in range(3)]
    releaser = threading.Thread(target=release)
    for t in (*workers, releaser):
        t.start()
    for t in workers:
        t.join()
    stop.set()
    releaser.join()
    assert not wrong
