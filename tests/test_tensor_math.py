"""CPU check of the tensor-core kernel's tables and integer arithmetic: every
output of two steps (16,384 outputs), put together from exact integer sums as
the kernel does, equals the oracle's stream, and every sum stays where fp32
holds it exactly."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "mrg8_gb300", "csrc")
P = 2147483647


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("native") / "check_tensor")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "native", "check_tensor.cpp"),
                    os.path.join(CSRC, "mrg8g_tables.cpp"), "-pthread"], check=True)
    return exe


def test_conversions_exhaustive(check):
    r = subprocess.run([check, "conv"], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and "bad=0" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("words", ["seeded", "zeros and p", "all p", "one"])
def test_block_products_give_the_stream(check, oracle, tmp_path, words):
    from oracle import pyoracle as po
    st = oracle.seed(13579)
    if words == "zeros and p":
        st[0], st[3], st[7] = 0, P, 0
    elif words == "all p":  # every sum is 0 mod p: the outputs are p
        st[:] = P
    elif words == "one":
        st[:] = 0
        st[7] = 1
    stream, _ = oracle.generate(st, 2 * 8192, po.U32)
    stream.tofile(tmp_path / "stream.bin")
    r = subprocess.run([check, str(tmp_path / "stream.bin"), *[str(int(v)) for v in st]], capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
