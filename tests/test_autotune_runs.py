"""The tuner's last word, on the CPU with a stand-in: the schemes' best candidates are compared by whole runs, since a
scheme whose steps start early in the tail of the step before takes less than the sum of its launches."""

from __future__ import annotations

import types

import pytest

from ac_fdtd_b200 import autotune


class FakeBatch:
    """A launched step takes ``launched[candidate]`` ms alone, ``in_runs[scheme]`` per step in a run."""

    launched = {("fused", 128, 16, 0): 0.107, ("fused", 128, 8, 0): 0.103, ("two_sweeps", 128, 8, 0): 0.100,
                ("two_sweeps", 256, 4, 0): 0.110}
    in_runs = {"fused": 0.091, "two_sweeps": 0.099}

    def __init__(self):
        self.clock, self.ms, self.steps, self.profiling, self.candidate = 0.0, 0.0, 0, False, None

    def run(self, n):
        if self.profiling:
            self.ms, self.steps = self.ms + n * self.launched[self.candidate], self.steps + n
        else:
            self.clock += 1e-3 * (n * self.in_runs[self.candidate[0]] + 0.02)      # the wait at a run's end

    def synchronize(self):
        pass

    def profile(self, on):
        self.profiling, self.ms, self.steps = on, 0.0 if on else self.ms, 0 if on else self.steps

    def profile_read(self):
        return self.ms, 0.0, self.steps


def test_runs_decide_between_the_schemes(monkeypatch):
    twin = FakeBatch()
    monkeypatch.setattr(autotune, "time", types.SimpleNamespace(perf_counter=lambda: twin.clock))

    def apply(fake, candidate):
        fake.candidate = candidate

    launched = autotune._race(twin, list(twin.launched), apply, steps=4, repeats=1, passes=2)
    winner, timings = autotune._final(twin, launched, apply)
    assert winner == ("fused", 128, 8, 0)                    # its scheme's best geometry
    assert timings[winner] == pytest.approx(0.091, rel=0.01)
    assert timings[("two_sweeps", 128, 8, 0)] == pytest.approx(0.099, rel=0.01)
    assert timings[("two_sweeps", 256, 4, 0)] == pytest.approx(0.110)


def test_a_single_scheme_is_not_timed_again():
    twin = FakeBatch()
    launched = {c: ms for c, ms in twin.launched.items() if c[0] == "fused"}
    winner, timings = autotune._final(twin, launched, lambda *_: pytest.fail("applied again"))
    assert winner == ("fused", 128, 8, 0) and timings == launched


def test_batch_candidates_hold_the_planes_that_untuned_batches_take():
    """An untuned batch takes 4 to 8 planes per tile of the fused step; tuned, it has to find one at least as good."""
    planes = {c[2] for c in autotune.BATCH_CANDIDATES if c[0] == "fused" and c[3] == 0}
    assert {4, 5, 6, 8} <= planes
