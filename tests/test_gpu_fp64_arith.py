"""The FP64 engine's arithmetic (sums and products as multiply-adds of registers, quotients that share
a denominator) rounds exactly like the plain IEEE operators: bit for bit on device-generated operands,
significands near all ones and near powers of two and signed zeros among them."""
import ctypes
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
    out = str(tmp_path_factory.mktemp("fp64arith") / "libfp64arith.so")
    subprocess.run([nvcc, "-std=c++17", "-O3", "-fmad=false", "-gencode", "arch=compute_103a,code=sm_103a", "-shared",
                    "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "cfd-2d-ns-fv_gb300", "csrc"),
                    os.path.join(HERE, "gpu_helpers", "fp64_arith_check.cu"), "-o", out], check=True, capture_output=True)
    lib = ctypes.CDLL(out)
    lib.arith_check.argtypes = [ctypes.c_ulonglong, ctypes.c_ulonglong] + [ctypes.c_int] * 4 + [
        ctypes.POINTER(ctypes.c_ulonglong)]
    return lib


@pytest.mark.parametrize("elo,ehi,ma,mb", [(-60, 60, 0, 0), (-3, 20, 0, 0), (-30, 30, 0, 1), (-30, 30, 1, 1),
                                           (-30, 30, 2, 0), (-30, 30, 0, 2), (-1, 1, 1, 2), (-30, 30, 3, 0),
                                           (-30, 30, 0, 3), (0, 0, 3, 3)])
def test_arithmetic_rounds_as_ieee(helper, elo, ehi, ma, mb):
    bad = (ctypes.c_ulonglong * 3)()
    for seed in (1, 2):
        assert helper.arith_check(1 << 26, seed * 104729 + elo * 31 + ma * 3 + mb, elo, ehi, ma, mb, bad) == 0
        assert list(bad) == [0, 0, 0], f"sums, products, quotients that differ: {list(bad)}"
