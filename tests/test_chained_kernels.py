"""Kernels that may start before the kernel ahead of them in the stream has ended (programmatic
dependent launches of the FP64 LU): a parameter that is __restrict__, or const __restrict__ above all,
lets the compiler read what the kernel ahead still writes through the non-coherent path or ahead of the
kernel's own wait.  No run shows whether a compiler does so, the declaration does."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pyvl_b200" / "csrc"


def _kernels():
    """name -> (parameters, body) of every __global__ function."""
    found = {}
    for path in sorted(CSRC.glob("*.cu*")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s+)?(\w+)\(([^)]*)\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            found[m.group(1)] = (m.group(2), text[m.end():end])
    return found


KERNELS = _kernels()
WAITING = sorted(k for k, (_, body) in KERNELS.items() if "grid_wait()" in body)


def test_the_chain_is_found():
    launched = set()
    text = (CSRC / "lu.cu").read_text()
    for m in re.finditer(r"launch_chained\((?:\(const void\*\))?(\w+)", text):
        launched.add(m.group(1))
    launched = {n.replace("_fn", "") for n in launched if n not in ("const", "fn")}
    assert launched and WAITING
    for name in launched:  # top_fn, apply_fn: chosen among one kernel's forms
        assert any(name in k for k in WAITING), name


@pytest.mark.parametrize("name", WAITING)
def test_no_restrict_parameter(name):
    assert "__restrict__" not in KERNELS[name][0]
