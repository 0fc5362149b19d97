"""The tensor-core bulk kernel against the oracle at the sizes where its steps,
quarters and blocks of threads end, and on outputs whose conversion takes the
general path (exact comparison: every output is an integer or its one rounding)."""
import numpy as np
import pytest

from mrg8_helpers import P, state_with_output
from oracle import pyoracle as po
from test_plain_gpu import KINDS, as_bytes, gen_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", KINDS)
def test_edges_of_steps(cuda, oracle, kind):
    import torch

    import mrg8_gb300 as m
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    step = 8192
    g = m.MRG8(99 + kind)
    for n in (1023, 1024, 2047, 2048, 2051, step - 1, step, step + 1, 3 * step + 2049, sms * step - 1, sms * step + 2,
              (3 * sms + 1) * step - 511):
        for offset in range(4):
            st = g.get_state()
            ref, end = oracle.generate(st, n, kind, nthreads=8)
            out = gen_device(g, n, kind, cuda, offset=offset)
            assert np.array_equal(as_bytes(out), as_bytes(ref)), (n, offset)
            assert np.array_equal(g.get_state(), end)


@pytest.mark.parametrize("at", [0, 65, 4000, 8191])
def test_outputs_of_the_general_conversion(cuda, oracle, at):
    """One output of a given residue, among them every edge of f64_fma_rare and
    f32_fma_rare and v = 0x7FFFFFBF in both scalings."""
    import mrg8_gb300 as m
    rng = np.random.default_rng(at)
    g = m.MRG8(1)
    residues = [0, 1, 2, 1 << 16, (1 << 17) - 1, 1 << 17, (1 << 17) + 1, (1 << 23) - 1, 1 << 23, (1 << 24) + 1,
                0x7FFF0000, 0x7FFF0001, 0x7FFFFEFF, 0x7FFFFF00, 0x7FFFFF01, 0x7FFFFFBF, 0x7FFFFFC0, P - 1]
    for r in residues:
        st = state_with_output(at, r, rng)
        for kind in KINDS:
            g.set_state(st)
            n = 9001
            ref, _ = oracle.generate(st, n, kind)
            out = gen_device(g, n, kind, cuda)
            assert np.array_equal(as_bytes(out), as_bytes(ref)), (r, kind)


@pytest.mark.parametrize("kind", KINDS)
def test_host_calls_around_the_mapped_buffer(cuda, oracle, kind):
    """Host calls on both sides of the largest that the kernel writes into mapped
    memory (128 KB), in turn on one handle."""
    import mrg8_gb300 as m
    g = m.MRG8(5 + kind)
    full = (128 << 10) // po.KIND_DTYPE[kind]().itemsize
    for n in (1, full, full + 1, 3, full - 1, 1023, 1024, 2 * full, 1):
        st = g.get_state()
        ref, end = oracle.generate(st, n, kind)
        host = np.full(n + 2, 3, dtype=po.KIND_DTYPE[kind])
        g._generate(host, n, kind)
        assert np.array_equal(host[:n].view(np.uint8), ref.view(np.uint8)), n
        assert (host[n:] == 3).all() and np.array_equal(g.get_state(), end)
