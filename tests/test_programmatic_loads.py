"""Kernels launched with programmatic stream serialisation become resident while
the kernel before them still writes.  Read-only loads (__ldg, const __restrict__)
promise the compiler memory that does not change while the kernel runs, and it
may take them ahead of the wait, so a source file with such launches has none."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "cloning-lbm-mpi_gb300" / "csrc"
SOURCES = [p for p in sorted(CSRC.glob("*.cu")) if "ProgrammaticStreamSerialization" in p.read_text()]


def code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def test_there_are_such_sources():
    assert {"clbm_step.cu", "clbm_refops.cu"} <= {p.name for p in SOURCES}


@pytest.mark.parametrize("name", [p.name for p in SOURCES] + ["clbm_physics.cuh", "clbm_reseed.cuh", "clbm_common.cuh"])
def test_no_read_only_loads(name):
    text = code(CSRC / name)
    assert "__ldg" not in text and "ld.global.nc" not in text
    assert not re.search(r"\bconst\b[^;,(){}]*\*\s*__restrict__", text)
