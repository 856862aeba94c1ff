"""The tensor memory's instructions want all lanes of a warp at the same place (``.sync.aligned``).  A GPU cannot show that a kernel keeps to
this: the compiler may bring lanes together again where the source does not, until it does not.  So the sources are read: on the way from a
wait, a branch, a loop's head or a barrier to such an instruction the warp has to be brought together (``warp_whole``,
``warp_all`` of csrc/common.cuh), unless the line says that the branch is the same for all lanes ("uniform")."""
import importlib
import os
import re

import pytest

build = importlib.import_module("daisi-llogos_b200.csrc.build")
CSRC = os.path.dirname(build.__file__)

PARTS = re.compile(r"\b(if|for|while|else|break|continue|return)\b|mbar_wait\(|__syncthreads\(|bar\.sync|cluster_barrier\(")
JOINS = re.compile(r"\bwarp_(whole|all)\(")
WANTS = re.compile(r"\btmem_(ld|st)\d+\(|tcgen05\.(alloc|dealloc)\.")
REGISTERS = re.compile(r"^\s*for \(int \w+ = 0; [^;]+; \+\+\w+\) [^{]*;\s*$")      # one statement over a thread's own values


def lines_that_want_the_warp(text):
    """(line number, line, whether the warp is whole there) of every call that wants all of its lanes."""
    found, whole = [], False
    for number, line in enumerate(text.splitlines(), 1):
        code, _, comment = line.partition("//")
        if "__device__" in code or "__global__" in code:
            whole = False
            continue
        uniform = "uniform" in comment
        splits = PARTS.search(code) and not uniform and not (REGISTERS.match(code) and not re.search(r"\bif\b|mbar_wait", code))
        if WANTS.search(code):
            found.append((number, line.strip(), whole and not splits))
        if JOINS.search(code):
            whole = True
        elif splits:
            whole = False
    return found


@pytest.mark.parametrize("source", ["gemm_tc.cu", "attention_tc.cu"])
def test_the_warp_is_whole_where_tensor_memory_wants_it(source):
    with open(os.path.join(CSRC, source)) as f:
        found = lines_that_want_the_warp(f.read())
    assert len(found) >= 8, found
    assert not [f for f in found if not f[2]]


def test_the_reading_finds_what_it_looks_for():
    wrong = "__device__ void f() {\n  warp_whole();\n  tmem_ld16(a, r);\n  if (row < n) {\n    out[row] = 1;\n  }\n  tmem_ld16(b, r);\n}"
    assert [w for _, _, w in lines_that_want_the_warp(wrong)] == [True, False]
    right = wrong.replace("  tmem_ld16(b", "  warp_whole();\n  tmem_ld16(b")
    assert [w for _, _, w in lines_that_want_the_warp(right)] == [True, True]
