"""Closing a room cut over several GPUs, on the CPU with stand-in parts: a neighbour's GPU stores into a
part's ghost planes, and a closed part's memory goes to the next solver of its GPU, so every part is
waited for before the first is closed; parts on one GPU need no such wait."""

from __future__ import annotations

import re
from pathlib import Path

import pytest

from ac_fdtd_b200.slabs import SlabGroup

NATIVE = Path(__file__).resolve().parents[1] / "ac_fdtd_b200" / "csrc" / "acfdtd_b200.cu"


class FakePart:
    def __init__(self, name, calls):
        self.name, self.calls = name, calls
        self.solver = self

    def synchronize(self):
        self.calls.append(("wait", self.name))

    def close(self):
        self.calls.append(("close", self.name))


@pytest.mark.parametrize("several", [True, False])
def test_parts_on_several_gpus_are_all_waited_for_first(several):
    calls = []
    group = SlabGroup.__new__(SlabGroup)
    group.slabs = [FakePart(n, calls) for n in range(3)]
    group._several_devices = several
    group.close()
    waits = [("wait", n) for n in range(3)] if several else []
    assert calls == waits + [("close", n) for n in range(3)]


@pytest.mark.parametrize("runner, events", [("run_fused_slabs", "done_ev"), ("run_slabs_impl", "pres_done")])
def test_a_parts_own_stream_ends_after_its_neighbours_last_stores(runner, events):
    """Callers of the C interface close parts by themselves: each stream waits, after the step loop, for the
    neighbours' last stores (two GPUs are needed to run it)."""
    text = NATIVE.read_text()
    body = text[text.index(f"int {runner}("):]
    body = body[:body.index("\n}\n")]
    loop = body.rindex("for (int64_t t = 0; t < n_steps; t++)")
    assert re.search(rf"wait_for_ghost_stores\(parts, n, {events}, streams\);", body[loop:])
