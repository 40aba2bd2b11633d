"""Build the CUDA library in-tree: ``python -m ac_fdtd_b200.build``.

One shared object, ``libacfdtd_b200.so``, compiled by nvcc for sm_100a only: each source to an
object of its own (in parallel, only where it or a header is newer), then linked. ``-fmad=false``
keeps every multiply and add separately rounded, which is what lets the sweeps reproduce the
NumPy reference bit for bit (the reference's C backend uses ``-ffp-contract=off`` for the same
reason, ac-fdtd ``src/ac_fdtd/c_backend.py:15-18,41``).
"""

from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PACKAGE = Path(__file__).resolve().parent
ROOT = PACKAGE.parent
CSRC = PACKAGE / "csrc"
_SHARED = [CSRC / "acfdtd_device.cuh", CSRC / "acfdtd_host.cuh", CSRC / "acfdtd_resident.cuh",
           CSRC / "acfdtd_fused.cuh", CSRC / "acfdtd_adjoint.cuh", CSRC / "acfdtd_shell.cuh", ROOT / "include" / "acfdtd_b200.h"]
#: Every source with the headers it includes.
SOURCES = {CSRC / "acfdtd_b200.cu": _SHARED,
           CSRC / "acfdtd_fused.cu": [*_SHARED, CSRC / "acfdtd_pack.cuh", CSRC / "acfdtd_fused_kernel.cuh"],
           CSRC / "acfdtd_fused_batch.cu": [*_SHARED, CSRC / "acfdtd_pack.cuh", CSRC / "acfdtd_fused_kernel.cuh"],
           CSRC / "acfdtd_adjoint.cu": [*_SHARED, CSRC / "acfdtd_pack.cuh"],
           CSRC / "acfdtd_shell.cu": [CSRC / "acfdtd_shell.cuh", CSRC / "acfdtd_host.cuh",
                                      ROOT / "include" / "acfdtd_b200.h"],
           CSRC / "acfdtd_post.cu": [CSRC / "acfdtd_host.cuh", ROOT / "include" / "acfdtd_b200.h"]}
for _part in ("resident_f32", "resident_f64"):
    SOURCES[CSRC / f"acfdtd_{_part}.cu"] = [*_SHARED, CSRC / "acfdtd_pack.cuh", CSRC / "acfdtd_resident_kernel.cuh"]
OBJECTS = PACKAGE / "_build"
TARGET = PACKAGE / "libacfdtd_b200.so"

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17", "-fmad=false",
    "-Xcompiler", "-fPIC",
    "-I", str(ROOT / "include"),
]


def nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(found).exists():
        raise RuntimeError("nvcc not found; the CUDA library cannot be built")
    return found


def needs_build(target: Path = TARGET) -> bool:
    if not target.exists():
        return True
    newest = max(p.stat().st_mtime for source, headers in SOURCES.items() for p in (source, *headers))
    return target.stat().st_mtime < newest


def _run(command) -> str:
    result = subprocess.run(list(map(str, command)), capture_output=True, text=True)
    if result.returncode != 0:
        raise RuntimeError(f"nvcc failed:\n{' '.join(map(str, command))}\n{result.stdout}\n{result.stderr}")
    return result.stderr


def _compile(source: Path, force: bool, verbose: bool) -> Path:
    target = OBJECTS / (source.stem + ".o")
    newest = max(p.stat().st_mtime for p in (source, *SOURCES[source]))
    if not force and target.exists() and target.stat().st_mtime >= newest:
        return target
    tmp = target.with_suffix(f".tmp{os.getpid()}.o")
    report = _run([nvcc(), *(["-Xptxas=-v"] if verbose else []), *NVCC_FLAGS, "-c", source, "-o", tmp])
    if verbose:
        sys.stderr.write(report)
    tmp.replace(target)
    return target


def build(force: bool = False, verbose: bool = False) -> Path:
    if not force and not needs_build():
        return TARGET
    OBJECTS.mkdir(exist_ok=True)
    with ThreadPoolExecutor(len(SOURCES)) as pool:
        objects = list(pool.map(lambda source: _compile(source, force, verbose), SOURCES))
    tmp = TARGET.with_suffix(f".tmp{os.getpid()}.so")
    _run([nvcc(), *NVCC_FLAGS, "-shared", *objects, "-o", tmp])
    tmp.replace(TARGET)
    return TARGET


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
