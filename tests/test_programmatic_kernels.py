"""Kernels launched as programmatic dependents are resident while the kernel before them still writes its
results, so their pointers to what kernels write are not __restrict__ const: the compiler may read through
such a pointer by the read-only path, whose data must not change while a kernel is resident."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "cfd-2d-ns-fv_gb300", "csrc")
MESH_ONLY = {"inc", "nbr"}   # what no kernel writes


def kernels(name):
    """(name, source) of every __global__ function of a file, comments removed."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    for m in re.finditer(r"__global__[^;{]*?\b(k\w+)\s*\(", src):
        depth, i = 0, src.index("{", m.end())
        for j in range(i, len(src)):
            depth += (src[j] == "{") - (src[j] == "}")
            if depth == 0:
                break
        yield m.group(1), src[m.start():j + 1]


@pytest.mark.parametrize("name,waits,expected", [
    ("fv2d_tiled.cuh", "pdl_wait()", {"k_tfirst"}),
    ("fv2d_kernels.cuh", "Prior()", {"k_gradient", "k_face", "k_face_pair", "k_update"}),
])
def test_no_read_only_pointers_to_written_arrays(name, waits, expected):
    found = {k: body for k, body in kernels(name) if waits in body}
    assert set(found) == expected
    for k, body in found.items():
        restricted = set(re.findall(r"__restrict__\s+(\w+)", body))
        assert restricted <= MESH_ONLY, f"{k}: {restricted - MESH_ONLY}"
