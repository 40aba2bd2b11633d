"""Steps that are launched early (programmatic dependents) are resident while the step before still
writes the state, and the read-only load path is for data that nothing writes during a kernel. So
the sources of those steps may take that path only for what the host alone writes: layer profiles,
wall pairs, and the descriptions of a batch's rooms. (Such a load cannot be caught going wrong by its
outputs, which depend on the compiler's order and on what L1 happens to hold.)"""

from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "ac_fdtd_b200" / "csrc"
EARLY = ["acfdtd_adjoint.cu", "acfdtd_fused.cu", "acfdtd_fused_batch.cu", "acfdtd_fused_kernel.cuh"]
HOST_WRITTEN = re.compile(r"s\.(cell|face)\[\d\]( \+ .*)?$|profile \+ .*$|entry( \+ 1)?$|(from|h) \+ w$")
READ_ONLY = re.compile(r"(?:__ldg|\bldg|ld\.global\.nc)\w*\s*\(")


def _argument(text, start):
    depth = 1
    for at in range(start, len(text)):
        depth += {"(": 1, ")": -1}.get(text[at], 0)
        if depth == 0:
            return text[start:at]
    raise ValueError("unbalanced call")


@pytest.mark.parametrize("name", EARLY)
def test_read_only_loads_are_of_host_written_data(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for match in READ_ONLY.finditer(text):
        argument = _argument(text, match.end()).strip()
        assert HOST_WRITTEN.match(argument), f"{name}: read-only load of {argument}"
    assert "__restrict__" not in text        # from which the compiler may choose that path itself


def test_every_early_launch_is_in_those_sources():
    found = {p.name for p in CSRC.iterdir() if "launch_after(" in p.read_text()}
    assert found <= {*EARLY, "acfdtd_host.cuh"}
