"""mrg8g_generate_host with a pointer to device memory in place of a host buffer: small
calls, which the host copies itself, treat it as large ones do (the copy engine either
takes it or refuses it with a status), and never touch it from the host."""
import ctypes as C

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def test_device_pointer(cuda, oracle):
    import torch

    import mrg8_gb300 as m
    lib = m.load()
    seen = []
    for n in (100_000, 1, 1000, 16384):
        g = m.MRG8(9)
        st = g.get_state()
        buf = torch.zeros(n, dtype=torch.float64, device=cuda)
        rc = lib.mrg8g_generate_host(g.handle, C.c_void_p(buf.data_ptr()), n, po.F64_ORIGINAL)
        torch.cuda.synchronize()
        seen.append(rc)
        want, end = oracle.generate(st, n, po.F64_ORIGINAL)
        if rc == 0:
            assert np.array_equal(buf.cpu().numpy(), want) and np.array_equal(g.get_state(), end)
        else:
            assert not bool(buf.any()) and np.array_equal(g.get_state(), st)
    assert len(set(seen)) == 1, seen


def test_pinned_memory(cuda, oracle):
    import torch

    import mrg8_gb300 as m
    for n in (1, 1000, 20_000):
        g = m.MRG8(10)
        st = g.get_state()
        out = torch.empty(n, dtype=torch.float64, pin_memory=True)
        g.rand(out)
        want, _ = oracle.generate(st, n, po.F64_ORIGINAL)
        assert np.array_equal(out.numpy(), want)
