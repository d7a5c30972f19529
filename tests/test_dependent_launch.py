"""Kernels started as programmatic dependent launches wait for the kernel before them.

A kernel that launch() starts may be placed on the GPU while its predecessor still runs; only the
wait at its head orders the two, so the sources are checked for it.
"""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pulsesuite_gb300" / "csrc"
SOURCES = {p.name: p.read_text() for p in sorted(CSRC.glob("*.cu*"))}


def _close(s, i):
    depth = 0
    for j in range(i, len(s)):
        depth += {"(": 1, ")": -1}.get(s[j], 0)
        if depth == 0:
            return j
    raise AssertionError("unbalanced parentheses")


def _bodies():
    """name -> [first statement of the body] of every __global__ definition"""
    out = {}
    for text in SOURCES.values():
        for m in re.finditer(r"__global__", text):
            k = re.compile(r"\b(k_\w+)\s*\(").search(text, m.end())
            rest = text[_close(text, k.end() - 1) + 1:].lstrip()
            if rest.startswith("{"):
                out.setdefault(k.group(1), []).append(rest[1:].lstrip().split(";")[0])
    return out


BODIES = _bodies()
# launched by name, or through a pointer set from names in the line before
LAUNCHED = sorted({m.group(1) for text in SOURCES.values()
                   for m in re.finditer(r"\blaunch\((?:\w+::)?(k_\w+)", text)} | {"k_tc_gemm"})


@pytest.mark.parametrize("kernel", LAUNCHED)
def test_waits_first(kernel):
    assert BODIES[kernel] == ["pdl_enter()"] * len(BODIES[kernel])


def test_every_dependent_launch_is_seen():
    calls = sum(len(re.findall(r"\blaunch\(", t)) for n, t in SOURCES.items() if n != "launch.cuh")
    named = sum(len(re.findall(r"\blaunch\((?:(?:\w+::)?k_|kernel\b)", t)) for t in SOURCES.values())
    assert LAUNCHED and calls == named
