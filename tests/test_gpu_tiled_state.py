"""The FP32 engine's inside: which kernels a step takes (so that tests which compare them compare what they say),
and in batches: a kernel that gave up (a copy or a barrier that timed out, a refused descriptor) leaves its
tiles at different stages; every call that returns results reports it."""
import ctypes
import glob
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def helper(tmp_path_factory, pkg):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path_factory.mktemp("tiledstate") / "libtiledstate.so")
    rest = [o for o in glob.glob(os.path.join(pkg.build.BUILD, "*.o")) if not o.endswith("fv2d_tiled.cu.o")]
    cmd, = [cmd for src, cmd in pkg.build._units() if src == "fv2d_tiled.cu"]   # as the library's own unit
    subprocess.run(cmd + ["-shared", os.path.join(HERE, "gpu_helpers", "tiled_state_check.cu"), *rest, "-o", out],
                   check=True, capture_output=True)
    return ctypes.CDLL(out)


def mesh_case(pkg, **opt):
    mg = pkg.meshgen
    case = dict(mg.DEFAULT_CASE, u=mg.mach_speed(0.5), BC1="SLIP_WALL", BC2="FREESTREAM", CFL=0.5, **opt)
    return pkg.fv2d._Desc(mg.channel_bump_quads(24, 12)), pkg.case_from_dict(case)


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("bits,words", [(0, ""), (2, "tile copies"), (4, "descriptor"), (8, "barrier"), (12, "descriptor")])
def test_kernel_errors_reach_the_caller(pkg, helper, bits, words, order):
    d, cs = mesh_case(pkg, solution_poly_order=order)
    rc = [ctypes.c_int() for _ in range(3)]
    msg = ctypes.create_string_buffer(256)
    assert helper.batch_with_error(ctypes.byref(d.desc), ctypes.byref(cs), bits, *[ctypes.byref(r) for r in rc], msg, 256) == 0
    assert [bool(r.value) for r in rc] == [bits != 0] * 3
    assert len({r.value for r in rc}) == 1 and words in msg.value.decode()


@pytest.mark.parametrize("kind,size,order,path", [
    ("quads", (5, 4), 1, 2), ("quads", (139, 70), 1, 2), ("bump", 9000, 1, 2), ("bump", 76000, 1, 2), ("bump", 84000, 1, 3),
    ("bump", 130000, 1, 0), ("quads", (5, 4), 0, 1), ("bump", 9000, 0, 1)])
def test_kernels_of_a_solve(pkg, helper, kind, size, order, path):
    mg = pkg.meshgen
    grid = mg.channel_bump_quads(*size) if kind == "quads" else mg.voronoi_bump_channel(size, seed=3)
    d = pkg.fv2d._Desc(grid)
    _, cs = mesh_case(pkg, solution_poly_order=order)
    assert helper.solver_path(ctypes.byref(d.desc), ctypes.byref(cs)) == path


@pytest.mark.parametrize("orders,path", [((1,), 2), ((1, 0), 2), ((0, 0), 1), ((0, 1, 1), 2)])
def test_kernels_of_a_batch(pkg, helper, orders, path):
    d, _ = mesh_case(pkg)
    cases = (pkg.Case * len(orders))(*[mesh_case(pkg, solution_poly_order=o)[1] for o in orders])
    assert helper.batch_path(ctypes.byref(d.desc), cases, len(orders)) == path
