"""Bulk calls (which may overlap the kernel before them on a stream) inside a captured
graph, behind nodes of every kind: copies, memsets, other kernels, a second stream's
work through events, and a batch; replays equal the oracle."""
import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def test_behind_other_nodes(cuda, oracle):
    import torch

    import mrg8_gb300 as m
    g, h = m.MRG8(21), m.MRG8(22)
    n, k = 200_003, 500
    x = torch.empty(n, dtype=torch.float64, device=cuda)
    y = torch.empty(n, dtype=torch.int32, device=cuda)
    z = torch.empty(k, dtype=torch.float64, device=cuda)
    src = torch.arange(n, dtype=torch.float64, device=cuda)
    outs = [torch.empty(4000, dtype=torch.float32, device=cuda) for _ in range(8)]
    plans = [m.Batch([(m.seed_state(50 + i), 3, o, po.F32_SHIFTED) for i, o in enumerate(outs)], use_graph=False,
                     blocks_per_sm=cap) for cap in (0, 2)]
    for p in plans:  # set-up outside the capture
        p.launch()
    side = torch.cuda.Stream()
    seen = []

    def calls():
        x.zero_()                       # memset or fill
        g.rand(x[1:5000])
        x.copy_(src)                    # device copy
        g.rand(x[:n - 1])
        seen.append(x.clone())
        here = torch.cuda.current_stream()
        side.wait_stream(here)
        with torch.cuda.stream(side):   # first node of the side stream
            h.randint(y)
            h.rand(z)
        g.rand(x[:k])                   # beside it
        here.wait_stream(side)
        g.rand(x[k:2000])               # behind both
        x[:k].add_(z)
        for p in plans:
            for o in outs:
                o.zero_()
            p.launch()
            g.rand(x[3000:5001])
        y.add_(1)

    states = [g.get_state(), h.get_state()]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    st, sh = states
    first = np.arange(n, dtype=np.float64)
    _, st = oracle.generate(st, 4999, po.F64_ORIGINAL)
    first[:n - 1], st = oracle.generate(st, n - 1, po.F64_ORIGINAL)
    wy, sh = oracle.generate(sh, n, po.U32)
    wz, sh = oracle.generate(sh, k, po.F64_ORIGINAL)
    last = first.copy()
    last[:k], st = oracle.generate(st, k, po.F64_ORIGINAL)
    last[k:2000], st = oracle.generate(st, 2000 - k, po.F64_ORIGINAL)
    last[:k] += wz
    for _ in plans:
        last[3000:5001], st = oracle.generate(st, 2001, po.F64_ORIGINAL)
    assert np.array_equal(g.get_state(), st) and np.array_equal(h.get_state(), sh)
    for _ in range(3):
        for t in (x, y, z, seen[0], *outs):
            t.fill_(7)
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(seen[0].cpu().numpy(), first)
        assert np.array_equal(x.cpu().numpy(), last)
        assert np.array_equal(y.cpu().numpy().view(np.uint32), (wy + np.uint32(1)).astype(np.uint32))
        for i, o in enumerate(outs):
            s = m.seed_state(50 + i)
            _, s = oracle.generate(s, 3, po.U32)
            want, _ = oracle.generate(s, 4000, po.F32_SHIFTED)
            assert np.array_equal(o.cpu().numpy(), want), i
    for p in plans:
        p.close()
