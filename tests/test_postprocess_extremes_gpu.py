"""Decay curves of signals whose energy is so small or so large that its reciprocal is not a normal
double, and of signals with infinities and NaN (on a GPU), at each split of a signal: one tile (up to
2048 samples), in registers, and in global memory. Against the host's sequential sums, which differ
by at most n eps relative in the sums (1e-9 dB, as for ordinary signals) -- and, where squares are
below the normal range, by the rounding of each square to a multiple of 5e-324."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import postprocess as device
from ac_fdtd_b200 import room as host

pytestmark = pytest.mark.gpu

SIZES = [600, 2048, 5000, 100_003]


def _signal(n):
    return np.random.default_rng(n).standard_normal(n) * np.exp(-9.0 * np.arange(n) / n)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("amplitude", [1e-151, 1e-156, 1e-157, 1e150, 3e151])
def test_very_quiet_and_very_loud(n, amplitude):
    x = amplitude * _signal(n)
    with np.errstate(under="ignore"):
        want = host.schroeder_decay(x)
    got = device.schroeder_decay(x)
    assert got[0] == 0.0 and np.all(got <= 1e-9)
    np.testing.assert_allclose(got, want, rtol=0.0, atol=1e-9)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_not_finite(n, value):
    x = _signal(n)
    x[n // 3] = value
    got = device.schroeder_decay(x)
    assert np.all(got == -120.0)        # the sum before it is not finite, so neither is any ratio

