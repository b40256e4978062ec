"""Kernels launched as programmatic dependents (those that call pdl_wait) run
while the kernel before them may still be writing the fields. Only tables that
no kernel of a step writes may be declared unaliased or read through the
read-only path in them."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "biofvm-b_b200" / "csrc"
TABLES = {"seg_start", "seg_voxel", "t1", "t2", "A", "B"}  # agents' segments and constants, bulk coefficients
TABLE_VIEWS = {"a", "b"}                                   # bulk_kernel's vector views of A and B


def kernels():
    for src in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", src.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
            depth, i = 1, m.end()
            while depth:  # the parameter list
                depth += {"(": 1, ")": -1}.get(text[i], 0)
                i += 1
            params, body0 = text[m.end():i - 1], text.index("{", i)
            depth, j = 1, body0 + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[j], 0)
                j += 1
            yield m.group(1), params, text[body0:j]


DEPENDENTS = [(n, p, b) for n, p, b in kernels() if "pdl_wait()" in b]


def test_the_dependents_are_found():
    names = {n for n, _, _ in DEPENDENTS}
    assert {"cells_kernel", "bulk_kernel", "sweep_strided_tma_kernel", "sweep_contig_pipe_kernel",
            "adjoint_dots_kernel", "adjoint_dots_flat_kernel", "cells_keep_kernel", "cells_adjoint_kernel",
            "adjoint_solve_strided_tma_kernel", "adjoint_solve_contig_pipe_kernel"} <= names


@pytest.mark.parametrize("name,params,body", DEPENDENTS, ids=[n for n, _, _ in DEPENDENTS])
def test_only_tables_are_read_only(name, params, body):
    unaliased = set(re.findall(r"__restrict__\s*(\w+)", params))
    assert unaliased <= TABLES, f"{name}: {sorted(unaliased - TABLES)}"
    local = set(re.findall(r"__restrict__\s*(\w+)", body)) - {"sm"}  # sm: the warp's shared memory
    assert not local, f"{name}: {sorted(local)}"
    read_only = set(re.findall(r"__ldg\(\s*(\w+)", body))
    assert read_only <= TABLES | TABLE_VIEWS, f"{name}: {sorted(read_only)}"
