"""Kernels launched as programmatic dependents (those that call pdl_wait) take nothing that the grid before
them writes through a const __restrict__ pointer: the compiler may read such a pointer with non-coherent
loads and move them over the wait.  Allowed are the caller's operands of a chain whose first kernel is
launched in plain stream order, and pointers read by ld_after_wait alone."""
import glob
import os
import re

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = sorted(glob.glob(os.path.join(REPO, "blas-for-multi-core-dsp_gb300", "csrc", "*.cu")))
ALLOWED = {("wdigits_kernel", "W"),         # the caller's operand, behind wexp_kernel
           ("stencil_rs_kernel", "src")}    # rs_walk: ld_after_wait


def _kernels(text):
    """(name, parameters, body) of every __global__ function of a source."""
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\([^{;]*?\)\s+)?(\w+)\(", text):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        j = text.index("{", i) + 1
        k, depth = j, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), text[m.end():i - 1], text[j:k]


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(p) for p in SOURCES])
def test_dependents_read_through_plain_pointers(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for name, params, body in _kernels(text):
        if "pdl_wait" not in body:
            continue
        found = re.findall(r"const \w+ \*\s*__restrict__ (\w+)", params)
        assert [p for p in found if (name, p) not in ALLOWED] == [], name


def test_every_dependent_is_found():
    names = {n for p in SOURCES for n, _, b in _kernels(re.sub(r"//[^\n]*", "", open(p).read())) if "pdl_wait" in b}
    assert {"wdigits_kernel", "thin_oz_kernel", "thin_oz_reduce_kernel", "thin_tc_kernel", "thin_tc_join_kernel",
            "stencil_rs_kernel", "slice_kernel", "ozaki_gemm_kernel", "ozaki_wide_kernel", "ozaki_join_kernel",
            "bf16x3_gemm_kernel"} <= names
