"""Rules that the CUDA sources keep, checked by reading them.

A kernel that raises bits of the error word may start some of its blocks when others have raised one already.  Where
its threads meet at barriers or in warp collectives, they have to take one decision on that word: a block that only
some of its threads left computes with what the leavers should have written.
"""
import glob
import os
import re
from functools import lru_cache

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "next_b200", "csrc")
BLOCK = re.compile(r"__syncthreads|cluster\.sync")
WARP = re.compile(r"__\w+_sync\(|__syncwarp")
LEAVES = re.compile(r"if \((?P<cond>[^{};]*\*err & kErrAbort[^{};]*)\)\s*(\{|return)")


def functions(path):
    """(name, is a kernel, body) of the functions defined in a source file."""
    src = re.sub(r"//[^\n]*", "", open(path).read())
    src = re.sub(r"__launch_bounds__\([^()]*\)", "", src)
    for m in re.finditer(r"\b(\w+)\s*\(([^;{}]*)\)\s*\{", src):
        head = src[max(src.rfind("}", 0, m.start()), src.rfind(";", 0, m.start())) + 1:m.start()]
        if m.group(1) in ("if", "for", "while", "switch", "return") or not re.search(r"__(global|device)__", head):
            continue
        depth, k = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            k += 1
        yield m.group(1), "__global__" in head, src[m.end():k]


def closure(pattern, bodies):
    """Names of the functions whose bodies match, or that call such a function."""
    names = {n for n, _, b in bodies if pattern.search(b)}
    while True:
        more = {n for n, _, b in bodies if n not in names and any(re.search(rf"\b{c}\b\s*(<[^;{{}}]*>)?\(", b) for c in names)}
        if not more:
            return names
        names |= more


@lru_cache(maxsize=1)
def sources():
    files = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
    return [f for path in files for f in functions(path)]


def test_sources_are_read():
    kernels = {n for n, kernel, _ in sources() if kernel}
    assert {"internal_kernel", "walk_group_kernel", "walk_reference_kernel", "cells_kernel"} <= kernels


@pytest.mark.parametrize("name", sorted({n for n, kernel, _ in sources() if kernel}))
def test_threads_that_meet_leave_together(name):
    every = sources()
    raising = closure(re.compile(r"\braise_error\("), every)
    block, warp = closure(BLOCK, every), closure(WARP, every)
    for n, kernel, body in every:
        if n != name or not kernel or n not in raising:
            continue
        for m in LEAVES.finditer(body):
            cond = m.group("cond")
            if n in block:
                assert "__syncthreads_or(" in cond, f"{n}: a block decides in parts ({cond})"
            elif n in warp:
                assert "__any_sync(0xffffffffu" in cond, f"{n}: a warp decides in parts ({cond})"
