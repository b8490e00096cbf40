"""Kernels whose roles may give up a wait hold no barrier without a bound in the loop of that wait: whoever left the loop would never come to it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc")
WAIT, BARRIER = re.compile(r"mbar_wait_(bounded|warp)\("), re.compile(r"bar\.sync|__syncthreads\(\)")


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _loops(code):
    """Bodies of the for and while loops in braces."""
    for m in re.finditer(r"\b(for|while)\s*\(", code):
        at, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(code[at], 0)
            at += 1
        while code[at].isspace():
            at += 1
        if code[at] != "{":
            continue
        start, depth = at, 0
        while True:
            depth += {"{": 1, "}": -1}.get(code[at], 0)
            at += 1
            if not depth:
                break
        yield code[start:at]


@pytest.mark.parametrize("path", [p for p in sorted(glob.glob(os.path.join(CSRC, "*.cu"))) if WAIT.search(_code(p))], ids=os.path.basename)
def test_no_barrier_without_a_bound_beside_a_wait(path):
    for body in _loops(_code(path)):
        assert not (WAIT.search(body) and BARRIER.search(body)), body[:400]
