"""Relative error of the FP64 reciprocal square roots (kernels.cuh) over two binades, measured on the device.

Tolerances: 2^-19 for the approximation instruction (20 significant bits, read and written); 2^-44 for the form of
the mixed far field, what one Newton step on an FP32 seed (2^-22.9) gives; 2^-51 for FP64 results (a few
rounding errors)."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import PKG, ROOT

pytestmark = pytest.mark.gpu


def test_errors(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "rsqrt_error")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-ftz=true",
                    "-I", os.path.join(PKG, "csrc"), os.path.join(ROOT, "tests", "cpp", "rsqrt_error.cu"), "-o", exe],
                   check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    seed, mixed, full = map(float, out.split())
    print("2^-x: seed %s" % out.strip())
    assert seed < 2.0 ** -19 and mixed < 2.0 ** -44 and full < 2.0 ** -51, out
