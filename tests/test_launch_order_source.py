"""Kernels are launched so that their blocks may be placed before the previous
kernel of the stream has completed; each waits on the device before it touches
memory.  The read-only data path (``ld.global.nc``: ``__ldg``, or a load
through a ``const __restrict__`` pointer) promises data that is constant for
the kernel's whole lifetime, and the cache-hint intrinsics are loads that the
compiler may move, so neither is held behind that wait.  An earlier kernel's
results must therefore be read by ordinary loads or by volatile asm."""
from __future__ import annotations

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "aerial-mimo-tc-optimization_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))


def _code(path):
    """The file without its comments."""
    text = open(path).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f) for f in FILES])
def test_no_read_only_path_loads(path):
    found = re.findall(r"__restrict__|__ldg|__ldc[agsv]|__ldlu|ld\.global\.nc", _code(path))
    assert not found, f"{os.path.basename(path)}: {sorted(set(found))}"


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f) for f in FILES])
def test_every_kernel_waits_before_its_first_access(path):
    """wait_previous() stands in each kernel before any branch, loop or pointer read of its body."""
    code = _code(path)
    for m in re.finditer(r"__global__", code):
        name = re.search(r"(\w+)\s*\((?!\()", code[m.end():].split("__launch_bounds__", 1)[-1].split(")", 1)[1]).group(1)
        body = code[code.index("{", m.end()):]
        at = body.find("wait_previous();")
        assert at >= 0, name
        assert not re.search(r"\b(if|for|while|switch|return)\b|\[[^\]\d]", body[:at]), name
