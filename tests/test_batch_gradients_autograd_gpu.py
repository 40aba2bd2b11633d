"""Gradients of batches against autograd through a plain float64 leapfrog (the one that ``perf/cases.py`` checks
outputs with, none of this package's kernels), on a GPU: rooms with whole and ragged rows, one-cell axes and rows of
one chunk, with and without a layer and air. Bounds as for single rooms (60 steps of some 30 roundings, forward and
back, of values up to the largest): 1e-9 in double and 2e-4 in single precision, 2e-3 there for the sums over a wall."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200.adjoint import DifferentiableBatch

pytestmark = pytest.mark.gpu

STEPS = 60
SHAPES = [(13, 11, 24), (1, 9, 4), (12, 4, 6), (7, 1, 5), (20, 17, 15), (6, 8, 1)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("layer, air", [(0, False), (2, False), (0, True), (2, True)])
def test_gradients_of_batches(layer, air, dtype):
    torch = pytest.importorskip("torch")
    from perf import cases

    described, specs = [], []
    for shape in SHAPES:
        rng = np.random.default_rng([*shape, layer])
        d = cases._description(rng, shape, STEPS, walls=True, layer=layer, layer_faces=2, air=air, receivers=2, dx=0.02)
        described.append((d, rng.standard_normal((2, STEPS))))
        specs.append(cases._objects(d))
    batch = DifferentiableBatch(specs, dtype=dtype, max_steps=STEPS)
    for r, (d, _) in enumerate(described):
        batch.batch.add_volume_source(r, cases._metres(d, d["source"]), d["signal"])
        for cell in d["receivers"]:
            batch.batch.add_pressure_receiver(r, cases._metres(d, cell))
    recorded = batch.forward(STEPS)
    wanted = [cases._gradients(d, target) for d, target in described]
    found = batch.backward([want[0].cpu().numpy() - target for want, (_, target) in zip(wanted, described)])
    value, total = (1e-9, 1e-9) if dtype == np.float64 else (2e-4, 2e-3)

    def close(got, want, bound, what):
        want = np.asarray(want.detach().cpu() if isinstance(want, torch.Tensor) else want, dtype=np.float64)
        error = np.max(np.abs(np.asarray(got, dtype=np.float64) - want)) / np.max(np.abs(want))
        assert error <= bound, f"{what}: {error:.3e}"

    for r, (forward, g, walls, cells) in enumerate(wanted):
        close(recorded[r], forward, value, f"room {r}: recordings")
        close(found[r].signal[0], g[0], value, f"room {r}: dL/dsignal")
        close(found[r].walls, walls, total, f"room {r}: dL/dxi")
        scale = max(float(c.abs().max()) for c in cells)
        for got, want in zip(found[r].wall_cells, cells, strict=True):
            assert np.max(np.abs(got - want.detach().cpu().numpy())) <= value * scale
    batch.batch.close()
