"""Kernels that start while the one before still runs (griddepcontrol.wait) read the arrays of a solve
by plain loads: a non-coherent load is only allowed on memory that nothing writes while the kernel lives,
and the compiler may move it above the wait. The sources are read for it: __ldg and const __restrict__
are for what no kernel of the chain writes, the topology's tables, the right-hand side of the whole solve
and the residual checks."""
import os
import re

import pytest

from conftest import ROOT

FIXED = {"nb8", "nb", "k", "table", "counts", "g", "rhs", "rhat", "check"}  # k, nb: rows of the tables; g: of the records


def _functions(name):
    """(name, parameters, body) of the functions defined in a source file."""
    with open(os.path.join(ROOT, "hnanosolver_b200", "csrc", name)) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    for m in re.finditer(r"\b(\w+)\(([^;{}]*)\)\s*\{", src):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
        yield m.group(1), m.group(2), src[m.end():i]


@pytest.mark.parametrize("name", ["hns_multigrid.cu", "hns_rbgs_split.cu"])
def test_arrays_of_the_solve_are_read_by_plain_loads(name):
    found = 0
    for fn, params, body in _functions(name):
        if "griddepcontrol.wait" not in body:
            continue
        found += 1
        read = re.findall(r"(?:__ldg|ld8|ldf4)\((?:reinterpret_cast<[^>]*>\()?\s*(\w+)", body)
        restricted = re.findall(r"\bconst\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)
        assert set(read) | set(restricted) <= FIXED, (fn, read, restricted)
    assert found >= 2


@pytest.mark.parametrize("name", ["hns_rows.cuh", "hns_advance.cu", "hns_fire.cu", "hns_mixed.cu", "hns_adjoint.cu"])
def test_arrays_that_a_kernel_writes_are_read_by_plain_loads(name):
    """In-place kernels: a pointer that is not const is not given to a load that is __ldg inside."""
    loads = r"(?<!\w)(?:__ldg|vload|sload|ld3|ld_half4|vel_z|(?:vel|scalar)_row<\w+>|vel_half_row)\((?:reinterpret_cast<[^>]*>\()?\s*(\w+)"
    found = 0
    for fn, params, body in _functions(name):
        if "__global__" not in params and "kernel" not in fn + params:
            continue
        found += 1
        pointers = re.findall(r"(const\s+)?[\w:]+\s*\*\s*(?:__restrict__\s+)?(\w+)", params)
        written = {p for const, p in pointers if not const}
        assert not written & set(re.findall(loads, body)), (fn, params[:120])
    assert found
