"""Kernels that may start while the kernel in front of them still runs must not read through the read-only
path, nor through pointers that promise no alias: both promises hold for a kernel's whole lifetime, which
begins before the wait for the kernel in front, and let the compiler move a load ahead of that wait."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "f2k_cuda_b200" / "csrc"


def _kernels(source):
    """(name, text from __global__ to the closing brace) of every kernel of a source file."""
    source = re.sub(r"//[^\n]*", "", source)
    for m in re.finditer(r"__global__", source):
        brace = source.index("{", m.start())
        depth, end = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(source[end], 0)
            end += 1
        yield re.search(r"(\w+)\s*\(", source[:brace][m.start():].split("__launch_bounds__", 1)[-1].split(")", 1)[1]).group(1), \
            source[m.start():end]


WAITING = [(f.name, name, text) for f in sorted(CSRC.glob("*.cu")) for name, text in _kernels(f.read_text())
           if "griddepcontrol.wait" in text or "grid_dependency_wait" in text]


def test_the_waiting_kernels_are_found():
    assert {n for _, n, _ in WAITING} == {"attn_fwd_sm100_kernel", "qk_prologue_kernel", "rmsnorm_rows128_kernel",
                                         "rope4_rows128_kernel"}


@pytest.mark.parametrize("file,name,text", WAITING, ids=[n for _, n, _ in WAITING])
def test_no_read_only_loads(file, name, text):
    for word in ("__ldg", "__restrict__", "ld.global.nc"):
        assert word not in text, f"{file}: {name} uses {word}"
