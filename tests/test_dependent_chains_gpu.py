"""Chains of dependent launches through the persistent kernels, and captured
scans with two predecessors.

Every launch may be set up while the kernel ahead of it still runs, and some read
ahead of their wait (prefetches; reduce-then-scan from its second launch on). Here
each step reads what the step before has just written, at sizes where the kernels
with units, the persistent select, the L2-buffered scan and several
reduce-then-scan chunks run; the grids are checked, so that the chain cannot lose a
kernel to another dispatch. Exact against the oracle.
"""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu

TILE = 4096


def _dev(x):
    return torch.from_numpy(x.view(np.int32)).cuda()


@pytest.mark.parametrize("captured", [False, True])
def test_chain_through_the_persistent_kernels(cuda, captured):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 4 * 5 * sms * TILE + 3  # 3041 tiles; reduce-then-scan: 3 chunks
    few = 7 * sms * TILE + 1    # below the kernel with units, above one tile per CTA when that is off
    rng = np.random.default_rng(n)
    x = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    offs = np.unique(np.concatenate([[0, n], rng.integers(0, n, size=50)])).astype(np.uint64)
    d, d_off = _dev(x), _dev(offs.astype(np.uint32))
    bufs = [torch.empty(n + 1, dtype=torch.int32, device="cuda") for _ in range(8)]
    flags = torch.empty(n, dtype=torch.uint8, device="cuda")
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()
    with Plan("csdl", "u32", max_n=n) as plan, Plan("rts", "u32", max_n=n) as rts, \
            Plan("csdl", "u32", max_n=few) as low:
        low.set_mid_max(0)
        b = [t[:n] for t in bufs]

        def grid(p, size, want):
            assert p.geometry(size)["grid"] == want

        def chain():
            plan.scan(d, out=b[0], inclusive=True, stream=side)
            grid(plan, n, sms)
            plan.scan_segmented(b[0], d_off, out=b[1], stream=side)
            grid(plan, n, sms)
            rts.scan(b[1], out=b[2], inclusive=True, stream=side)
            assert rts.geometry(n)["launches"] == 4
            plan.scan(b[2], out=bufs[3][1:], stream=side)  # off a 16-byte boundary
            grid(plan, n, sms)
            rts.scan(bufs[3][1:], out=b[4], stream=side)
            plan.scan(b[4], out=b[4], inclusive=True, stream=side)
            low.scan(b[4][:few], out=b[4][:few], stream=side)
            grid(low, few, min(sms, (few + 4 * TILE - 1) // (4 * TILE)))
            torch.ge(b[4], 0, out=flags.view(torch.bool))
            plan.select(b[4], flags, out=b[5], num_selected=count, stream=side)
            grid(plan, n, sms)
            rts.scan(b[4], out=b[6], stream=side)
            rts.scan(b[6], out=b[6], inclusive=True, stream=side)
            plan.scan(b[6], out=b[7], inclusive=True, stream=side)

        graph = None
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            if captured:
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=side):
                    chain()
            for k in range(3):
                d.copy_(_dev(np.roll(x, k)))
                for t in bufs:
                    t.fill_(-1)
                for _ in range(3):
                    graph.replay() if graph else chain()
        side.synchronize()
        for p in (plan, rts, low):
            p.check(side)
    a = oracle.segscan(oracle.scan(np.roll(x, 2), True), offs, False)
    a = oracle.scan(oracle.scan(oracle.scan(a, True), False), False)
    a = oracle.scan(a, True)
    a[:few] = oracle.scan(a[:few], False)
    assert np.array_equal(b[4].cpu().numpy().view(np.uint32), a)
    sel = a[a.view(np.int32) >= 0]
    assert int(count.item()) == sel.size
    assert np.array_equal(b[5].cpu().numpy().view(np.uint32)[:sel.size], sel)
    a = oracle.scan(oracle.scan(a, False), True)
    assert np.array_equal(b[6].cpu().numpy().view(np.uint32), a)
    assert np.array_equal(b[7].cpu().numpy().view(np.uint32), oracle.scan(a, True))


@pytest.mark.parametrize("n", [70_001, 2_000_003, 3100 * TILE + 9])
def test_captured_scans_that_join_two_streams(cuda, n):
    # A scan on each of two streams, then a join: the next launch has a kernel on
    # its own stream and an event of the other ahead of it, and reads both results.
    rng = np.random.default_rng(n)
    x = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    flags = (rng.random(n) < 0.3).astype(np.uint8)
    d, d_flags = _dev(x), torch.from_numpy(flags).cuda()
    a, b, c, e = (torch.empty_like(d) for _ in range(4))
    f = torch.empty_like(d_flags)
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    main, other = torch.cuda.Stream(), torch.cuda.Stream()
    with Plan("csdl", "u32", max_n=n) as p, Plan("csdl", "u32", max_n=n) as q, Plan("rts", "u32", max_n=n) as r:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            other.wait_stream(main)
            p.scan(d, out=a, inclusive=True, stream=main)
            q.scan(d, out=b, stream=other)
            with torch.cuda.stream(other):
                f.copy_(d_flags)
            main.wait_stream(other)
            p.select(b, f, out=c, num_selected=count, stream=main)  # of the other stream's scan
            other.wait_stream(main)
            q.scan(a, out=b, inclusive=True, stream=other)
            r.scan(a, out=e, inclusive=True, stream=main)
            main.wait_stream(other)
            r.scan(b, out=a, stream=main)
        for k in range(3):
            y = np.roll(x, 5 * k)
            d.copy_(_dev(y))
            for t in (a, b, c, e):
                t.fill_(-1)
            torch.cuda.synchronize()
            graph.replay()
            graph.replay()
            torch.cuda.synchronize()
            incl = oracle.scan(y, True)
            sel = oracle.scan(y, False)[flags != 0]
            assert int(count.item()) == sel.size
            assert np.array_equal(c.cpu().numpy().view(np.uint32)[:sel.size], sel)
            twice = oracle.scan(incl, True)
            assert np.array_equal(e.cpu().numpy().view(np.uint32), twice)
            assert np.array_equal(b.cpu().numpy().view(np.uint32), twice)
            assert np.array_equal(a.cpu().numpy().view(np.uint32), oracle.scan(twice, False))
        for plan in (p, q, r):
            plan.check()
