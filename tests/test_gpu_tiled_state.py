"""FP32 batches: a kernel that gave up (a copy or a barrier that timed out, a refused descriptor) leaves its
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
