"""CPU check of the rule that names a batch launch's kernel and blocks."""
import os
import subprocess

from conftest import ROOT


def test_rule(tmp_path):
    from mrg8_gb300 import build
    exe = str(tmp_path / "check_batch_kernel")
    subprocess.run([build.nvcc(), "-O1", "-std=c++17", "-I" + os.path.join(ROOT, "mrg8_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "check_batch_kernel.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
