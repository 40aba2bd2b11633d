"""The tuner on rooms that runs hold on chip, on the CPU with a stand-in solver: schemes whose runs take many steps
per launch count with the time of such a run, not of their launched step."""

from __future__ import annotations

import types

import numpy as np
import pytest

from ac_fdtd_b200 import autotune, solver as solver_module


class FakeSolver:
    """A launched step takes ``launched[scheme]`` ms; runs of the schemes in ``held`` take that per step."""

    launched = {"staged": 0.007, "fused": 0.008, "two_sweeps": 0.010}
    held = {}
    clock = 0.0

    def __init__(self, *_args, steps_per_graph=64, **_kwargs):
        self.p = np.zeros((4, 4, 4))
        self.steps_per_graph = steps_per_graph
        self.scheme, self.profiling, self.launches, self.ms, self.steps = "two_sweeps", False, 0, 0.0, 0

    def set_scheme(self, scheme):
        self.scheme = scheme

    def set_launch(self, *geometry):
        self.geometry = geometry

    set_staging = set_launch

    def run(self, n):
        is_held = self.scheme in self.held and n >= 8 and self.steps_per_graph and not self.profiling
        ms = n * (self.held if is_held else self.launched)[self.scheme]
        self.launches += 2 if is_held else n
        self.ms, self.steps = self.ms + ms, self.steps + n
        FakeSolver.clock += 1e-3 * ms

    def profile(self, on):
        self.profiling = on
        if on:
            self.ms, self.steps = 0.0, 0

    def profile_read(self):
        return self.ms, 0.0, self.steps

    def launch_count(self):
        return self.launches

    def synchronize(self):
        pass

    def close(self):
        pass


def _tuned(monkeypatch, held, steps_per_graph=64):
    monkeypatch.setattr(solver_module, "CudaAcousticFDTD", FakeSolver)
    monkeypatch.setattr(FakeSolver, "held", held)
    monkeypatch.setattr(autotune, "time", types.SimpleNamespace(perf_counter=lambda: FakeSolver.clock))
    solver = types.SimpleNamespace(grid=None, medium=None, courant=1.0, dtype=None, walls=None, absorbing_layer=None,
                                   air_absorption=None, steps_per_graph=steps_per_graph)
    return autotune.tune(solver, candidates=((64, 4), (128, 4)), staged_candidates=((2, 3, 32, 4),))


def test_held_rooms_keep_the_scheme_that_is_held(monkeypatch):
    winner, timings = _tuned(monkeypatch, {"fused": 0.002, "two_sweeps": 0.002})
    assert winner[0] == "fused"              # the faster launched step of the two that tie
    assert timings[winner] == pytest.approx(0.002)
    assert timings[("staged", 2, 3, 32, 4)] == pytest.approx(0.007)


def test_other_rooms_are_timed_launch_by_launch(monkeypatch):
    winner, timings = _tuned(monkeypatch, {})
    assert winner == ("staged", 2, 3, 32, 4) and timings[("two_sweeps", 64, 4)] == pytest.approx(0.010)


def test_a_solver_that_launches_step_by_step_gets_its_best_step(monkeypatch):
    winner, _ = _tuned(monkeypatch, {"fused": 0.002, "two_sweeps": 0.002}, steps_per_graph=0)
    assert winner[0] == "staged"
