"""Batches of one kind, each with a kernel of its own, and of mixed kinds: many uneven
instances with unaligned starts sharing steps, small batches and launches with few
resident blocks (the recurrence kernel), and outputs that the conversions leave to
their general path.  Every output against the oracle, exactly."""
import ctypes as C

import numpy as np
import pytest

from mrg8_helpers import state_with_output
from oracle import pyoracle as po
from test_batch_gpu import KINDS, as_bytes, check_canaries, expected, tdt
from test_dispatch_edges_gpu import EDGES

pytestmark = pytest.mark.gpu

MIXED = -1


def instances(cuda, rng, kind, lengths, offsets=True):
    import torch

    import mrg8_gb300 as m
    insts, meta = [], []
    for i, n in enumerate(lengths):
        k = KINDS[int(rng.integers(0, 5))] if kind == MIXED else kind
        off = int(rng.integers(0, 2**63)) if offsets and i % 3 == 0 else int(rng.integers(0, 10))
        lead = i % 4
        buf = torch.full((n + lead + 3,), -5, dtype=tdt(k), device=cuda)
        st = m.seed_state(int(rng.integers(0, 2**32)))
        insts.append((st, off, buf[lead:lead + n], k))
        meta.append((st, off, n, k, buf, lead))
    return insts, meta


def check(oracle, insts, meta, what):
    import torch
    torch.cuda.synchronize()
    for (st, off, n, kind, buf, lead), (_, _, view, _) in zip(meta, insts):
        want = expected(oracle, st, off, n, kind)
        assert np.array_equal(as_bytes(view), want.view(np.uint8)), (what, off, n, kind, lead)
        view.fill_(-5)
    check_canaries(meta)


def uneven(rng, count, max_log2):
    return [int(2 ** rng.uniform(0, max_log2)) if i % 7 else int(rng.choice([0, 1, 2, 3, 5, 7, 8, 9, 31, 129]))
            for i in range(count)]


@pytest.mark.parametrize("kind", KINDS + [MIXED])
def test_uneven_instances(cuda, oracle, kind):
    import mrg8_gb300 as m
    rng = np.random.default_rng(50 + kind)
    insts, meta = instances(cuda, rng, kind, uneven(rng, 130, 16) + [2047, 2048, 2049, 8191, 8193, 70001])
    for tile_rows, tiling in ((0, 0), (16, 1), (24, 0), (128, 1)):
        b = m.Batch(insts, tile_rows=tile_rows, tiling=tiling)
        b.launch()
        check(oracle, insts, meta, (tile_rows, tiling))
        b.close()


@pytest.mark.parametrize("longest", [512, 513, 1024, 1025])
@pytest.mark.parametrize("kind", KINDS + [MIXED])
def test_small_instances(cuda, oracle, kind, longest):
    """On both sides of the lengths at which the kernel changes."""
    import mrg8_gb300 as m
    rng = np.random.default_rng(900 + kind)
    lengths = [longest, longest - 1, 1, 0, 63, 64, 65, 511] + [int(v) for v in rng.integers(0, longest + 1, 60)]
    insts, meta = instances(cuda, rng, kind, lengths)
    for tiling in (0, 1):
        b = m.Batch(insts, tiling=tiling)
        b.launch()
        b.launch()
        check(oracle, insts, meta, tiling)
        b.close()


@pytest.mark.parametrize("kind", [po.U32, po.F64_ORIGINAL, MIXED])
def test_more_small_instances_than_resident_warps(cuda, oracle, kind):
    import torch

    import mrg8_gb300 as m
    rng = np.random.default_rng(77)
    warps = 9 * 4 * torch.cuda.get_device_properties(cuda).multi_processor_count
    for count in (warps - 1, warps + 1500):
        insts, meta = instances(cuda, rng, kind, [20 + i % 5 for i in range(count)], offsets=False)
        b = m.Batch(insts)
        b.launch()
        check(oracle, insts, meta, count)
        b.close()


@pytest.mark.parametrize("threads,blocks_per_sm", [(0, 1), (128, 2), (256, 1), (256, 100)])
@pytest.mark.parametrize("kind", KINDS + [MIXED])
def test_few_resident_blocks(cuda, oracle, kind, threads, blocks_per_sm):
    import mrg8_gb300 as m
    rng = np.random.default_rng(600 + kind)
    insts, meta = instances(cuda, rng, kind, uneven(rng, 60, 17) + [300001])
    for tile_rows, tiling in ((8, 1), (0, 0)):
        b = m.Batch(insts, tile_rows=tile_rows, threads=threads, blocks_per_sm=blocks_per_sm, tiling=tiling)
        assert b.config["blocks_per_sm"] == blocks_per_sm
        b.launch()
        b.launch()
        check(oracle, insts, meta, (tile_rows, tiling))
        b.close()


@pytest.mark.parametrize("kind", KINDS + [MIXED])
def test_no_alloc(cuda, oracle, kind):
    import torch

    import mrg8_gb300 as m
    from mrg8_gb300 import _lib as L
    lib = m.load()
    rng = np.random.default_rng(40 + kind)
    for lengths in (uneven(rng, 60, 17), [int(v) for v in rng.integers(0, 500, 200)], [200003, 65536, 3]):
        insts, meta = instances(cuda, rng, kind, lengths)
        arr = (L.Instance * len(insts))()
        for a, (st, off, out, k) in zip(arr, insts):
            a.state[:] = [int(v) for v in st]
            a.offset, a.n, a.out, a.kind = off, out.numel(), out.data_ptr() if out.numel() else 0, k
        stream = torch.cuda.current_stream().cuda_stream
        assert lib.mrg8g_batch_generate_noalloc(arr, len(insts), C.c_void_p(stream)) == 0, lib.mrg8g_last_error()
        check(oracle, insts, meta, len(lengths))


@pytest.mark.parametrize("kind", KINDS + [MIXED])
def test_edges_of_the_conversions(cuda, oracle, kind):
    """Batches whose outputs at a few places take every edge residue, as one kind and as
    mixed kinds (which make ORIGINAL of SHIFTED), on both kernels."""
    import torch

    import mrg8_gb300 as m
    rng = np.random.default_rng(8)
    insts, meta = [], []
    for r in sorted({v + d for v in EDGES for d in (0, 1)}):
        for at in (5, 300, 2100):
            for k in (KINDS if kind == MIXED else [kind]):
                n = at + 1 + int(rng.integers(0, 200))
                buf = torch.full((n + 3,), -5, dtype=tdt(k), device=cuda)
                st = state_with_output(at, r, rng)
                insts.append((st, 0, buf[:n], k))
                meta.append((st, 0, n, k, buf, 0))
    for blocks_per_sm in (0, 9):
        b = m.Batch(insts, blocks_per_sm=blocks_per_sm)
        b.launch()
        check(oracle, insts, meta, blocks_per_sm)
        b.close()
