"""Rooms held on chip by several threads at once, each on a stream of its own and beside other work (on a GPU): each
launch needs all its CTAs resident and waits for them, so launches of several rooms, each as large as the device
holds, must take their turns; the results are those of each room alone."""

from __future__ import annotations

import threading

import numpy as np
import pytest

from ac_fdtd_b200 import AirAbsorption, CudaAcousticFDTD, Grid, WallAdmittances

pytestmark = pytest.mark.gpu


def _solver(n, dtype, stream=0):
    solver = CudaAcousticFDTD(Grid(dx=0.03, nx=n, ny=n + 1, nz=n + 2), dtype=dtype, stream=stream,
                              walls=WallAdmittances.uniform(0.3), air_absorption=AirAbsorption())
    solver.add_volume_source((0.5, 0.6, 0.7), np.hanning(40))
    solver.add_pressure_receiver((0.3, 0.2, 0.2))
    return solver


def test_several_threads_and_streams():
    torch = pytest.importorskip("torch")
    rooms = [(70, np.float64), (80, np.float32), (72, np.float64), (93, np.float32)]
    runs = (9, 200, 8, 300)
    want = []
    for n, dtype in rooms:
        alone = _solver(n, dtype)
        alone.run(sum(runs))
        want.append((np.array(alone.p), alone.recorded_pressure))
        alone.close()
    failed = []

    def work(index):
        try:
            n, dtype = rooms[index]
            stream = torch.cuda.Stream(priority=-(index % 2))
            for _ in range(3):
                solver = _solver(n, dtype, stream.cuda_stream)
                before = solver.launch_count()
                for steps in runs:
                    solver.run(steps)
                assert solver.launch_count() - before == 2 * len(runs)
                solver.synchronize()
                np.testing.assert_array_equal(solver.p, want[index][0])
                np.testing.assert_array_equal(solver.recorded_pressure, want[index][1])
                solver.close()
        except BaseException as error:      # noqa: BLE001 (reported by the test's own thread)
            failed.append(error)

    busy = torch.randn(4096, 4096, device="cuda")
    threads = [threading.Thread(target=work, args=(index,)) for index in range(len(rooms))]
    side = torch.cuda.Stream()
    for t in threads:
        t.start()
    with torch.cuda.stream(side):
        while any(t.is_alive() for t in threads):
            for _ in range(4):
                busy = torch.tanh(busy @ busy)
            side.synchronize()
    for t in threads:
        t.join()
    assert not failed, failed[0]
