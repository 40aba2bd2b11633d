"""Adjoint gradients of single rooms against autograd through a plain float64 leapfrog (the one that
``perf/cases.py`` checks outputs with, none of this package's kernels), on a GPU: rooms so narrow in
y and z that a block of the adjoint step has fewer threads than there are air sums, or less than a
warp, and rooms with whole and ragged rows, with and without a layer.

In double precision the two differ by their order of summation: some 30 roundings per step forward
and back over 60 steps, 2 x 60 x 30 x 1.1e-16 = 4e-13 of the largest value, times up to a thousand
where a sum over all cells and steps cancels: 1e-9 with room to spare. In single precision (6e-8)
the same bound is 2e-4 for values and, with a factor of ten for the sums that cancel, 2e-3 for the
sums over the room (wall totals, air processes).
"""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200.adjoint import DifferentiableRoom

pytestmark = pytest.mark.gpu

STEPS = 60
NARROW = [(12, 4, 6), (9, 2, 4), (11, 1, 3), (30, 2, 2), (17, 3, 5), (8, 5, 1)]
WIDE = [(13, 11, 24), (20, 17, 15), (9, 6, 131)]


def _compare(shape, dtype, layer, air):
    torch = pytest.importorskip("torch")
    from perf import cases

    rng = np.random.default_rng([*shape, layer])
    d = cases._description(rng, shape, STEPS, walls=True, layer=layer, layer_faces=2, air=air, receivers=2, dx=0.02)
    target = rng.standard_normal((2, STEPS))
    recorded, g, walls, cells = cases._gradients(d, target)
    objects = cases._objects(d)
    room = DifferentiableRoom(objects.pop("grid"), dtype=dtype, **objects, max_steps=STEPS,
                              wrt=("signal", "walls", "air") if air else ("signal", "walls"))
    room.solver.add_volume_source(cases._metres(d, d["source"]), d["signal"])
    for cell in d["receivers"]:
        room.solver.add_pressure_receiver(cases._metres(d, cell))
    forward = room.forward(STEPS)
    found = room.backward(recorded.cpu().numpy() - target)

    value, total = (1e-9, 1e-9) if dtype == np.float64 else (2e-4, 2e-3)

    def close(got, want, bound, what):
        want = np.asarray(want.detach().cpu() if isinstance(want, torch.Tensor) else want, dtype=np.float64)
        error = np.max(np.abs(np.asarray(got, dtype=np.float64) - want)) / np.max(np.abs(want))
        assert error <= bound, f"{what}: {error:.3e}"

    close(forward, recorded, value, "recordings")
    close(found.signal[0], g[0], value, "dL/dsignal")
    close(found.initial_p, g[1], value, "dL/dp0")
    close(found.walls, walls, total, "dL/dxi")
    for got, want in zip(found.wall_cells, cells, strict=True):
        scale = max(float(c.abs().max()) for c in cells)
        assert np.max(np.abs(got - want.detach().cpu().numpy())) <= value * scale
    if air:
        strength, tau = (torch.as_tensor(x) for x in cases._processes(*d["air"], d["dt"]))
        close(found.strength * strength.numpy(), g[8].cpu() * strength, total, "dL/dlog strength")
        close(found.relaxation_time * tau.numpy(), g[9].cpu() * tau, total, "dL/dlog tau")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", NARROW)
def test_air_gradients_of_narrow_rooms(shape, dtype):
    _compare(shape, dtype, 0, True)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("shape", WIDE)
@pytest.mark.parametrize("layer, air", [(0, False), (2, False), (0, True), (2, True)])
def test_gradients_of_rooms(shape, layer, air, dtype):
    _compare(shape, dtype, layer, air)
