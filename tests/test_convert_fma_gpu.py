"""The conversions of the tensor-core kernels as compiled for the GPU (one fused
multiply-add of bit patterns, whose device and host bodies differ, and the general path
of the values that it leaves out) on every v in [0, 2^31 - 1], exactly."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_every_value(cuda, tmp_path):
    from mrg8_gb300 import build
    exe = str(tmp_path / "check_convert_gpu")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-I" + build.CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "native", "check_convert_gpu.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
