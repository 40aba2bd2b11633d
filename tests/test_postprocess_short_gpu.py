"""Short and middling signals (on a GPU): the decay kernels where a curve's runs per thread change (512 samples
for runs of one, 1024, 2048, 3072, 4096, 6144 and 12,288) and where fits and clarities change their number of CTAs
(20,000 samples in all parts for eight, 40,000 for four, 80,000 for two, fewer with many channels), against the
host's sequential sums: 1e-9, as sums of n terms in another order differ by at most n eps. Their time: one CTA
needs neither a cluster's launch nor its barriers, which cost more than the work on such signals."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from ac_fdtd_b200 import _native
from ac_fdtd_b200 import postprocess as device
from ac_fdtd_b200 import room as host

pytestmark = pytest.mark.gpu


def _signals(channels, n):
    rng = np.random.default_rng(n)
    rates = rng.uniform(9.0, 14.0, channels)[:, None]
    return rng.standard_normal((channels, n)) * np.exp(-rates * np.arange(n) / n)


@pytest.mark.parametrize("edge", [512, 1024, 2048, 3072, 4096, 6144, 12_288])
@pytest.mark.parametrize("beyond", [-1, 0, 1])
def test_curves_on_both_sides_of_each_run(edge, beyond):
    x = _signals(3, edge + beyond)
    got = device.schroeder_decay(x)
    np.testing.assert_allclose(got, host.schroeder_decay(x), rtol=0.0, atol=1e-9)
    assert np.all(got[:, 0] == 0.0)


@pytest.mark.parametrize("channels, n", [(2, 19_999), (2, 20_000), (18, 20_001), (19, 40_000), (19, 39_999),
                                         (38, 80_000), (75, 80_001), (2, 8193)])
def test_sums_on_both_sides_of_each_split(channels, n):
    x, rate = _signals(channels, n), n / 2.0
    for got, want in ((device.reverberation_time(x, rate), host.reverberation_time),
                      (device.early_decay_time(x, rate), host.early_decay_time)):
        np.testing.assert_allclose(got, [want(signal, rate) for signal in x], rtol=1e-9)
    np.testing.assert_allclose(device.clarity(x, rate, 0.05), [host.clarity(signal, rate, 0.05) for signal in x],
                               rtol=1e-9, atol=1e-9)


def _microseconds(torch, call, calls=100):
    for _ in range(5):
        call()
    torch.cuda.synchronize()
    graph, best = torch.cuda.CUDAGraph(), np.inf
    with torch.cuda.graph(graph):
        for _ in range(calls):
            call()
    for _ in range(5):
        start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        start.record()
        graph.replay()
        end.record()
        torch.cuda.synchronize()
        best = min(best, 1e3 * start.elapsed_time(end) / calls)
    return best


def test_short_signals_do_not_pay_for_clusters():
    """Against a clarity of 600 samples, which one launch's latency bounds (2.3 us): a curve of them 1.05 times as
    long (1.65 with a cluster's launch, barriers and long runs), a fit of 48 signals of 12,000 2.5 (4.4)."""
    torch = pytest.importorskip("torch")
    lib = _native.library()

    def times(channels, n):
        x = torch.as_tensor(_signals(channels, n), device="cuda")
        decay, out = torch.empty_like(x), torch.empty(channels, dtype=torch.float64, device="cuda")
        failed = torch.empty(channels, dtype=torch.int32, device="cuda")

        def stream():
            return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

        curve = _microseconds(torch, lambda: lib.acf_schroeder_decay(
            x.data_ptr(), channels, n, -120.0, decay.data_ptr(), stream()))
        fit = _microseconds(torch, lambda: lib.acf_decay_fit(
            decay.data_ptr(), channels, n, 48_000.0, -5.0, -35.0, out.data_ptr(), failed.data_ptr(), stream()))
        split = _microseconds(torch, lambda: lib.acf_clarity(
            x.data_ptr(), channels, n, n // 3, out.data_ptr(), stream()))
        return curve, fit, split

    short = times(48, 600)
    longer = times(48, 12_000)
    assert short[0] < 1.4 * short[2]
    assert longer[1] < 3.5 * short[2]
