"""Chains of scans without synchronisation, each reading what the one before
wrote: a launch that is set up early must not read its input, its
descriptors or its launch number before the kernel ahead has finished. Exact
against the oracle, eager and captured; other kernels (copies, fills, the
persistent scan, compaction) sit between the scans.
"""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu


def _dev(x):
    return torch.from_numpy(x.view({4: np.int32, 8: np.int64}[x.itemsize])).cuda()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("n", [5_000, 70_001, 600_000, 5_000_003])
def test_chain_of_scans(cuda, n, captured):
    rng = np.random.default_rng(n)
    x = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    offs = np.unique(np.concatenate([[0, n], rng.integers(0, n, size=50)])).astype(np.uint64)
    d, d_off = _dev(x), _dev(offs.astype(np.uint32))
    bufs = [torch.empty_like(d) for _ in range(7)]
    flags = torch.empty(n, dtype=torch.uint8, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()
    with Plan("csdl", "u32", max_n=n) as plan, Plan("rts", "u32", max_n=n) as rts:
        rts.set_small_max(0)

        def chain():
            plan.scan(d, out=bufs[0], inclusive=True, stream=side)
            plan.scan(bufs[0], out=bufs[1], stream=side)
            plan.scan_segmented(bufs[1], d_off, out=bufs[2], inclusive=True, stream=side)
            rts.scan(bufs[2], out=bufs[3], inclusive=True, stream=side)
            bufs[4].copy_(bufs[3])
            plan.scan(bufs[4], out=bufs[4], stream=side)
            torch.ge(bufs[4], 0, out=flags.view(torch.bool))
            plan.select(bufs[4], flags, out=bufs[5], num_selected=count, stream=side)
            plan.scan(bufs[4], out=bufs[6], inclusive=True, stream=side)

        graph = None
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=side):
                    chain()
            for k in range(3):
                d.copy_(_dev(np.roll(x, k)))
                for b in bufs:
                    b.fill_(-1)
                for _ in range(4):
                    graph.replay() if graph else chain()
        side.synchronize()
        plan.check(side)
    a = oracle.scan(oracle.scan(np.roll(x, 2), True), False)
    a = oracle.scan(oracle.segscan(a, offs, True), True)
    assert np.array_equal(bufs[3].cpu().numpy().view(np.uint32), a)
    a = oracle.scan(a, False)
    assert np.array_equal(bufs[4].cpu().numpy().view(np.uint32), a)
    sel = a[a.view(np.int32) >= 0]
    assert int(count.item()) == sel.size
    assert np.array_equal(bufs[5].cpu().numpy().view(np.uint32)[:sel.size], sel)
    assert np.array_equal(bufs[6].cpu().numpy().view(np.uint32), oracle.scan(a, True))
