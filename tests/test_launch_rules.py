"""What chained launches rely on, read from the CUDA sources.

A kernel launched with programmatic dependent launch starts while the kernel
before it still runs. Nothing it reads from that kernel may be loaded ahead
of its griddepcontrol.wait, and a const __restrict__ pointer lets the
compiler do just that (the load is invariant to it, a "memory" clobber does
not hold it back). So such pointers may only name what no kernel of a chain
writes: the mesh, the matrix and the maps between levels.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fvm_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))

# complete before a chain's first launch
CONSTANT = {
    "ci", "rowSlice", "c2fRow", "c2fCol",                                # maps between levels
    "ainv", "diag", "meta", "cols",                                      # matrix
    "row", "col", "w", "vol", "fc", "bFaces", "bIndexOfFace", "perm",    # mesh
    "coeff", "sec", "am", "source", "rhoVdt",                            # coefficients and fields of a step
    "pivots", "next",                                                    # elimination order, read by the host first
}


def text(name):
    s = open(os.path.join(CSRC, name)).read()
    s = re.sub(r"//[^\n]*", "", s)
    return re.sub(r"/\*.*?\*/", "", s, flags=re.S)


def block(s, at):
    """s from its first '{' after at to the matching '}'."""
    i = s.index("{", at)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(s[j], 0)
        j += 1
        if depth == 0:
            return s[i:j]


def kernels(name):
    """(kernel, parameters, body) of every __global__ function with a body."""
    s = text(name)
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(\w+)\(", s):
        depth, j = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(s[j], 0)
            j += 1
        if s[j:].lstrip().startswith("{"):
            yield m.group(1), s[m.end():j - 1], block(s, j)


def waits(body):
    return "FVM_PDL()" in body or "FVM_PDL_WAIT()" in body or "griddepcontrol.wait" in body


def restricted(params):
    return re.findall(r"__restrict__\s+(\w+)", params)


@pytest.mark.parametrize("name", SOURCES)
def test_only_constant_data_is_restrict_in_chained_kernels(name):
    bad = {}
    for k, params, body in kernels(name):
        extra = [p for p in restricted(params) if p not in CONSTANT] if waits(body) else []
        if extra:
            bad[k] = extra
    # what kernels inline: helpers and the accessors they gather through
    for m in re.finditer(r"__device__\s+__forceinline__\s+[\w ]+?(\w+)\(([^{;]*?)\)\s*(?:const\s*)?\{", text(name)):
        extra = [p for p in restricted(m.group(2)) if p not in CONSTANT]
        if extra:
            bad[m.group(1)] = extra
    for m in re.finditer(r"\bstruct\s+(\w+)\s*\{", text(name)):
        extra = [p for p in restricted(block(text(name), m.start())) if p not in CONSTANT]
        if extra:
            bad[m.group(1)] = extra
    assert not bad


def test_chained_launches_wait():
    waiting, others = set(), set()
    for name in SOURCES:
        for k, _, body in kernels(name):
            (waiting if waits(body) else others).add(k)
    assert waiting and others
    for name in SOURCES:
        for k in re.findall(r"pdl_launch(?:_smem)?\(\s*(k_\w+)", text(name)):
            assert k in waiting, f"{name}: {k} is launched ahead of its predecessor's end and does not wait"


def test_loop_control_ends_a_chain():
    """k_spmv_dot_pby_ell reads the search direction ahead of its wait: the
    update that wrote it is complete because the loop's test, launched after
    it, is not a dependent launch."""
    solver = text("solver.cu")
    for k in ("k_loop_init", "k_loop_check"):
        assert re.search(r"\b%s(?:<\w+>)?<<<" % k, solver)
        assert not re.search(r"pdl_launch(?:_smem)?\(\s*%s\b" % k, solver)
        assert not any(waits(body) for n, _, body in kernels("solver.cu") if n == k)
