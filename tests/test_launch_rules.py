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


def functions(name):
    """(name, body) of every function definition of a file, roughly: an
    identifier, a parameter list and a body."""
    s = text(name)
    for m in re.finditer(r"^[A-Za-z][^\n;#(){}=]*?([\w:~]+)\(", s, flags=re.M):
        depth, j = 1, m.end()
        while depth and j < len(s):
            depth += {"(": 1, ")": -1}.get(s[j], 0)
            j += 1
        if re.match(r"\s*(const\s*)?(:[^{;]*)?\{", s[j:]):
            yield m.group(1), block(s, j)


HOST = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cpp", ".hpp")))
COPIES = r"cudaMemset\(|cudaMemcpy\([^;]*cudaMemcpyHostToDevice|\bupload\("
# the arena's own members, and callers whose kernels run on the default stream
DEFAULT_STREAM = {"copy_h2d", "DeviceArena::copy_h2d", "upload", "CsrGraph", "fvm_csr_residual",
                  "fvm_learned_forward_csr", "fvm_learned_gradient_csr"}


@pytest.mark.parametrize("name", HOST)
def test_host_copies_end_before_another_stream_reads_them(name):
    """cudaMemcpy from pageable memory and cudaMemset are ordered before later
    work of the default stream only; level arrays, mesh arrays and network
    parameters are read on streams that do not wait for it. Whoever makes such
    a copy waits for the default stream (settle_device) after the last one."""
    s = text(name)
    checked = 0
    for fn, body in functions(name):
        at = [m.start() for m in re.finditer(COPIES, body)]
        checked += len(at)
        if at and fn not in DEFAULT_STREAM:
            assert "settle_device();" in body[at[-1]:], f"{name}: {fn}"
    if name.endswith(".cu"):
        assert checked == len(re.findall(COPIES, s))


def test_settle_waits_for_the_default_stream():
    assert "cudaStreamSynchronize(nullptr)" in dict(functions("solver.cu"))["settle_device"]


def test_host_build_ends_with_the_default_stream_empty():
    body = dict(functions("solver.cu"))["AmgHierarchy::build"]
    assert body.index("buildTail();") < body.index("settle_device();") < body.index("tunePlans();")
