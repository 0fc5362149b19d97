"""Bulk calls on both sides of the sizes at which they pass from the recurrence kernel
to the tensor cores, and outputs at the edges of the conversions' general path, against
the oracle (exact comparison: every output is an integer or its one rounding)."""
import numpy as np
import pytest

from mrg8_helpers import state_with_output
from test_plain_gpu import KINDS, as_bytes, gen_device

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", KINDS)
def test_sizes_around_the_change_of_kernel(cuda, oracle, kind):
    import mrg8_gb300 as m
    g = m.MRG8(700 + kind)
    for n in (895, 896, 897, 960, 1000, 1023, 1024, 1025, 1026, 1027):
        for offset in range(4):
            st = g.get_state()
            ref, end = oracle.generate(st, n, kind)
            out = gen_device(g, n, kind, cuda, offset=offset)
            assert np.array_equal(as_bytes(out), as_bytes(ref)), (n, offset)
            assert np.array_equal(g.get_state(), end)


# Values v that a conversion may leave out (f64_fma_rare: 23 leading ones; f32_fma_rare:
# below 1,280 and from 0x7FFFFC00 on) and their neighbours; v is the residue S or S - 1.
EDGES = [1, 1279, 1280, 0x7FFFFBFF, 0x7FFFFC00, (1 << 22) - 1, (1 << 23) - 1, 0xFFFFFD, 0xFFFFFE, 0x7FFFFDFF, 0x7FFFFE00,
         0x7FFFFEFF, 0x7FFFFF00, 0x7FFFFFBE, 0x7FFFFFBF, 0x7FFFFFC0]


@pytest.mark.parametrize("at", [3, 500, 1023, 8300])
def test_edges_of_the_conversions(cuda, oracle, at):
    import mrg8_gb300 as m
    rng = np.random.default_rng(at)
    g = m.MRG8(1)
    for r in sorted({v + d for v in EDGES for d in (0, 1)}):
        st = state_with_output(at, r, rng)
        for kind in KINDS:
            g.set_state(st)
            n = 9001
            ref, _ = oracle.generate(st, n, kind)
            out = gen_device(g, n, kind, cuda)
            assert np.array_equal(as_bytes(out), as_bytes(ref)), (r, kind)
