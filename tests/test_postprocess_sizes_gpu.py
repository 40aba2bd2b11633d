"""The decay kernels where their split of a signal changes: one CTA (sums up to 4096 samples, curves
in one tile up to 2048 and in registers up to 12,288), up to eight CTAs with the curve in registers
(98,304), curves scanned in global memory beyond, and parts that are ragged or empty; against the host's sequential FP64 sums. A sum of n terms in another order differs
by at most n eps relative (2.2e-16 n: 1e-10 at 450,000 samples), so curves are held to 1e-9 dB and
ratios and times to 1e-9."""

from __future__ import annotations

import numpy as np
import pytest

from ac_fdtd_b200 import postprocess as device
from ac_fdtd_b200 import room as host

pytestmark = pytest.mark.gpu


def _signals(channels, n):
    rng = np.random.default_rng(n)
    rates = rng.uniform(9.0, 14.0, channels)[:, None]
    return rng.standard_normal((channels, n)) * np.exp(-rates * np.arange(n) / n)


@pytest.mark.parametrize("n", [1, 2, 5, 511, 2048, 2049, 2071, 12_288, 12_289, 24_577, 98_303, 98_304, 98_305, 100_003, 450_007])
def test_curves_match_the_host(n):
    x = _signals(1 if n > 200_000 else 3, n)
    got = device.schroeder_decay(x)
    np.testing.assert_allclose(got, host.schroeder_decay(x), rtol=0.0, atol=1e-9)
    assert np.all(got[:, 0] == 0.0)


@pytest.mark.parametrize("n", [700, 4096, 4097, 16385, 100_003, 216_001, 450_007])
def test_times_and_clarity_match_the_host(n):
    rate = n / 2.0
    for signal in _signals(2, n):
        assert device.reverberation_time(signal, rate) == pytest.approx(host.reverberation_time(signal, rate), rel=1e-9)
        assert device.early_decay_time(signal, rate) == pytest.approx(host.early_decay_time(signal, rate), rel=1e-9)
        for split in (0.05, 0.08, 0.6):
            assert device.clarity(signal, rate, split) == pytest.approx(host.clarity(signal, rate, split), rel=1e-9)


def test_silence_and_many_channels():
    quiet = device.schroeder_decay(np.zeros((2, 5000)))
    assert np.all(quiet == -120.0)
    x = np.tile(_signals(1, 5000), (300, 1))
    got = device.schroeder_decay(x)
    assert np.all(got == got[0])            # every channel the same bits
