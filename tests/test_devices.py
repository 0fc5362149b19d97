"""CPU check of the per-device records: a host call keeps the address of its
device's record across stream waits while another thread may first use another
device, so a record must never move."""
import os
import subprocess

from conftest import ROOT


def test_records_keep_their_address(tmp_path):
    exe = str(tmp_path / "check_devices")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "mrg8_gb300", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "native", "check_devices.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
