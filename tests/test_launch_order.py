"""Kernels start while the kernel before them is still writing, and wait for it inside (griddepcontrol.wait). What they read
after the wait must not be readable before it: a pointer that promises the compiler unchanging memory (__restrict__, __ldg,
ld.global.nc) lets a load move across the wait. The sources are read here; no GPU is needed."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "damendaemon_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))
WEIGHTS = ("bias", "gamma", "beta", "weight", "weight2", "mu")          # no kernel writes these


def code(path):
    """The file without its comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_no_load_may_move_across_the_wait(path):
    text = code(path)
    assert "__restrict__" not in text
    assert "ld.global.nc" not in text
    for call in re.finditer(r"__ldg\((?:reinterpret_cast<[^>]*>\()?(?:p\.|a\.)?(\w+)", text):
        assert call.group(1) in WEIGHTS, call.group(0)


def test_every_kernel_waits():
    """Each kernel but the one that tests the limit of a wait, and those launched in plain order only."""
    without = []
    for path in SOURCES:
        text = code(path)
        starts = [m.start() for m in re.finditer(r"__global__", text)] + [len(text)]
        for a, b in zip(starts, starts[1:]):
            if "dd_grid_wait()" not in text[a:b]:
                without.append(re.search(r"(\w+_kernel)\s*\(", text[a:b]).group(1))
    assert without == ["wait_probe_kernel"]
