"""Kernels' bounded waits: what callers see once one has given up.  In processes of
their own, since the device's error word holds for the whole process."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def check(cuda, tmp_path_factory):
    from mrg8_gb300 import build
    objs = [os.path.join(build.BUILD, os.path.basename(s) + ".o") for s in build.sources()]
    if not all(os.path.exists(o) for o in objs):
        build.build(force=True)
    exe = str(tmp_path_factory.mktemp("native") / "check_waits")
    subprocess.run([build.nvcc(), *build.ARCH, "-O1", "-std=c++17", "-I" + build.INCLUDE, "-I" + build.CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "native", "check_waits.cpp"),
                    os.path.join(ROOT, "tests", "native", "short_waits.cu"), *objs], check=True)
    return exe


def test_a_wait_that_gives_up_ends_its_launch(check):
    r = subprocess.run([check, "kernel"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_every_call_reports_a_wait_that_gave_up(check):
    r = subprocess.run([check, "host"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
