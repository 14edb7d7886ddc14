"""The rule of dependent launches (csrc/common.cuh): a kernel that calls pdl_wait is resident while
its predecessor still writes, so what kernels of the chain write is never read through
__restrict__ pointers or __ldg, which promise that nothing else writes there meanwhile.  Read
from the sources: a load that the compiler moved above the wait shows in no result for certain.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "msbg-flip_b200",
                    "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
# block lists, offsets, the operator of the direct solve, and flags that kernels only raise
STATIC = {"tiles", "coarseOff", "Ainv", "cells", "slotOf", "list", "err", "errFlag"}


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _functions(src):
    """(signature, body) of every function with a body, kernels and device functions."""
    for m in re.finditer(r"__global__|__device__", src):
        i = min((src.find(c, m.start()) for c in "{;" if src.find(c, m.start()) >= 0))
        if src[i] == ";":
            continue
        depth, j = 0, i
        while True:
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            if not depth:
                break
            j += 1
        yield m.group(0), src[m.start():i], src[i:j]


def _dependent(name):
    return [(s, b) for kind, s, b in _functions(_code(name))
            if kind == "__global__" and "pdl_wait()" in b]


def test_the_dependent_kernels_are_found():
    found = sum(len(_dependent(f)) for f in FILES)
    assert found >= 14, found


@pytest.mark.parametrize("name", FILES)
def test_no_restrict_on_what_a_chain_writes(name):
    for sig, _ in _dependent(name):
        bad = set(re.findall(r"\*\s*__restrict__\s+(\w+)", sig)) - STATIC
        assert not bad, (sig, bad)


@pytest.mark.parametrize("name", FILES)
def test_helpers_of_dependent_kernels(name):
    # __ldg of the couplings alone; no __restrict__ in the device functions of these files that
    # take a vector of the chain
    if not _dependent(name) and name != "pressure_kernels.cuh":
        return
    src = _code(name)
    assert set(re.findall(r"__ldg\((\w+)\)", src)) <= {"pc"}
    for kind, sig, _ in _functions(src):
        if kind == "__device__":
            assert "__restrict__" not in sig, sig
