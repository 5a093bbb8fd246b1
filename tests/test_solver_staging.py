"""A solver's page-locked staging buffer holds every transfer that goes through it, on the smallest meshes
too, where the residual norm's partial sums are larger than any field."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

HERE = os.path.dirname(os.path.abspath(__file__))


def test_staging_buffer_holds_every_transfer(tmp_path):
    cxx = shutil.which("g++")
    inc = "/usr/local/cuda/include"
    if cxx is None or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no compiler or CUDA headers")
    exe = str(tmp_path / "staging_check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", inc, "-I", os.path.join(ROOT, "cfd-2d-ns-fv_gb300", "csrc"),
                    os.path.join(HERE, "cpu_helpers", "staging_check.cpp"), "-o", exe, "-L/usr/local/cuda/lib64", "-lcudart"],
                   check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(3, 3), (16, 8), (19, 8), (17, 9)])   # 9, 128, 152, 153 cells
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_residual_norm_of_small_meshes(pkg, nx, ny, precision):
    mg = pkg.meshgen
    case = dict(mg.DEFAULT_CASE, u=mg.mach_speed(0.5), BC1="SLIP_WALL", BC2="FREESTREAM", CFL=0.5)
    s = pkg.Solver(mg.channel_bump_quads(nx, ny), case, precision=getattr(pkg, precision))
    s.step(2)
    got = s.residual_norm()
    r = s.get(pkg.fv2d.F_RES).reshape(4, -1)
    # both sum squares in FP64: n rounded additions differ by at most n ulp
    np.testing.assert_allclose(got, np.sqrt((r * r).sum(axis=1)), rtol=2 * r.shape[1] * 2.3e-16, atol=0)
    s.close()
