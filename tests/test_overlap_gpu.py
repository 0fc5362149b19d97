"""Bulk calls that follow one another on a stream may overlap on the device; their
effects must not: readers between them see each call's outputs, the last writer
wins, and a captured sequence replays the same (exact against the oracle)."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

SIZES = [1000, 300_000, 5, 70_000, 300_001, 895, 2048]


def test_readers_between_calls(cuda, oracle):
    import torch

    import mrg8_gb300 as m
    g = m.MRG8(3)
    st = g.get_state()
    x = torch.empty(max(SIZES), dtype=torch.float64, device=cuda)
    seen = []
    for i in range(42):
        n = SIZES[i % len(SIZES)]
        g.rand(x[:n])
        seen.append(x[:n].clone())
    for i, v in enumerate(seen):
        want, st = oracle.generate(st, v.numel(), po.F64_ORIGINAL)
        assert np.array_equal(v.cpu().numpy(), want), i


def test_overwriting_calls_and_capture(cuda, oracle):
    import torch

    import mrg8_gb300 as m
    g = m.MRG8(4)
    n = 300_001
    x = torch.empty(n, dtype=torch.float64, device=cuda)

    def calls():
        g.rand(x)
        g.rand(x[:1000])
        g.rand(x[500:200_000])

    def expected(st):
        want, st = oracle.generate(st, n, po.F64_ORIGINAL)
        want[:1000], st = oracle.generate(st, 1000, po.F64_ORIGINAL)
        want[500:200_000], _ = oracle.generate(st, 199_500, po.F64_ORIGINAL)
        return want

    for _ in range(20):
        st = g.get_state()
        calls()
        assert np.array_equal(x.cpu().numpy(), expected(st))
    st = g.get_state()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    for _ in range(3):
        x.zero_()
        graph.replay()
        graph.replay()
        assert np.array_equal(x.cpu().numpy(), expected(st))
