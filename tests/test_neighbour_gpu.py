"""Bulk calls next to another library's kernels that use tensor memory and start
early (programmatic stream serialization), their blocks on the same SMs: one behind a
bulk call sees the call's outputs, one ahead of it still gets its tensor memory, and
all end."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def native(cuda, tmp_path_factory):
    from mrg8_gb300 import build
    so = str(tmp_path_factory.mktemp("native") / "tmem_neighbour.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", so,
                    os.path.join(ROOT, "tests", "native", "tmem_neighbour.cu")], check=True)
    lib = C.CDLL(so)
    lib.behind.argtypes = [C.c_void_p, C.c_void_p, C.c_uint32, C.c_int, C.c_void_p]
    lib.ahead.argtypes = [C.c_uint32, C.c_void_p, C.c_int, C.c_void_p]
    return lib


@pytest.mark.parametrize("n", [5, 300, 1000, 100_003, 3_000_001])
def test_kernels_around_bulk_calls(cuda, oracle, native, n):
    import torch

    import mrg8_gb300 as m
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    rounds, g = 12, m.MRG8(17)
    st = g.get_state()
    x = torch.empty(n, dtype=torch.float64, device=cuda)
    seen = torch.zeros((rounds, n), dtype=torch.float64, device=cuda)
    done = torch.zeros(1, dtype=torch.int32, device=cuda)
    stream = torch.cuda.current_stream().cuda_stream
    for r in range(rounds):
        assert native.ahead(20, done.data_ptr(), 2 * sms, stream) == 0
        g.rand(x)
        assert native.behind(x.data_ptr(), seen[r].data_ptr(), n, 4 * sms, stream) == 0
    torch.cuda.synchronize()
    assert int(done) == rounds * 2 * sms
    for r in range(rounds):
        want, st = oracle.generate(st, n, po.F64_ORIGINAL, nthreads=8)
        assert np.array_equal(seen[r].cpu().numpy(), want), r
