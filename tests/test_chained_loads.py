"""Kernels launched by launch_chained may be resident while the kernel before
them is still writing, so what earlier kernels write may not be read as data
that stays constant over the whole kernel: no `const T *__restrict__` and no
__ldg (the compiler may use read-only loads, and move them before the wait of
chain_begin).  Mesh inputs are constant for the whole build."""
import os
import re

import pytest

from conftest import ROOT

INPUTS = {"pts", "tris"}  # the caller's vertex and index arrays
CSRC = os.path.join(ROOT, "gpu-svo_b200", "csrc")


def _strip(text):
    return re.sub(r"//[^\n]*", "", text)


def _functions(text):
    """Top-level definitions of a source file (the code's layout: a definition
    starts in column 0, its body ends with a brace in column 0)."""
    return re.findall(r"^(?:template[^\n]*\n)?[A-Za-z_][^;{}]*?\([^;{]*?\)\s*(?:const\s*)?\{.*?^\}", text, flags=re.M | re.S)


def _constant_reads(fn):
    names = re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", fn)
    names += re.findall(r"__ldg\(\s*(?:\w+\.)?(\w+)", fn)
    return [n for n in names if n not in INPUTS]


def _chained(fns):
    """The chained kernels and every function of the file that they call."""
    names = {re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", f)).group(1): f for f in fns}
    reach = {n for n, f in names.items() if "__global__" in f and "chain_begin()" in f}
    grown = True
    while grown:
        more = {n for n in names if n not in reach and any(re.search(r"\b%s\s*(<[^;()]*>)?\s*\(" % n, names[r]) for r in reach)}
        reach |= more
        grown = bool(more)
    return {n: names[n] for n in reach}


@pytest.mark.parametrize("source", ["svo_voxelize.cu", "svo_octree.cu"])
def test_no_constant_reads_of_earlier_kernels_output(source):
    with open(os.path.join(CSRC, source)) as f:
        chained = _chained(_functions(_strip(f.read())))
    assert len(chained) >= 8
    bad = {n: r for n, f in chained.items() if (r := _constant_reads(f))}
    assert not bad


def test_every_chained_launch_is_of_a_kernel_that_waits():
    text = ""
    for source in ("svo_voxelize.cu", "svo_octree.cu"):
        with open(os.path.join(CSRC, source)) as f:
            text += _strip(f.read())
    launched = set(re.findall(r"launch_chained\((\w+)", text))
    assert launched
    kernels = {re.search(r"\b(k_\w+)\s*\(", f).group(1): f for f in _functions(text) if "__global__" in f}
    for k in launched:
        body = kernels[k][kernels[k].index("{") :]
        first = [s.strip() for s in re.sub(r"__shared__[^;]*;", "", body[1:]).split(";") if s.strip()][0]
        assert first == "chain_begin()", (k, first)
