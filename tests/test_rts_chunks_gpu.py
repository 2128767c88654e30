"""Reduce-then-scan at the edges of its split: one range of at most 2 tiles for
each of 5 CTAs per SM makes a chunk, and every launch reduces one chunk and
propagates the one before. Bit-exact against the oracle, on aligned buffers,
on views, in place, and with inputs that change between graph replays.
"""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu

NP = {"u32": np.uint32, "u64": np.uint64}
SIGNED = {4: np.int32, 8: np.int64}


def _rand(dtype, n, seed):
    return np.random.default_rng(seed).integers(0, np.iinfo(NP[dtype]).max, size=n, dtype=NP[dtype], endpoint=True)


def _dev(x):
    return torch.from_numpy(x.view(SIGNED[x.itemsize])).cuda()


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_sizes_around_ranges_and_chunks(cuda, dtype, off):
    tile = 16384 // np.dtype(NP[dtype]).itemsize
    ranges = 5 * torch.cuda.get_device_properties(0).multi_processor_count
    sizes = [5 * tile + 3, ranges * tile - off, ranges * tile + 1, 2 * ranges * tile - 1, 2 * ranges * tile + 1,
             4 * ranges * tile, 4 * ranges * tile + 7, 6 * ranges * tile + tile + 5]
    with Plan("rts", dtype, max_n=max(sizes)) as plan:
        plan.set_small_max(0)
        for k, n in enumerate(sizes):
            x = _rand(dtype, n, seed=n)
            inclusive = bool(k & 1)
            want = oracle.scan(x, inclusive)
            src = _dev(np.concatenate([np.zeros(off, NP[dtype]), x]))[off:]
            out = torch.full((n + 8,), -3, dtype=src.dtype, device="cuda")
            plan.scan(src, out=out[4:4 + n], inclusive=inclusive, n=n)
            got = out.cpu().numpy()
            assert np.array_equal(got[4:4 + n].view(NP[dtype]), want), n
            assert np.all(got[:4] == -3) and np.all(got[4 + n:] == -3), n
            plan.scan(src, out=src, inclusive=inclusive)  # in place
            assert np.array_equal(src.cpu().numpy().view(NP[dtype]), want), n
        plan.check()


def test_back_to_back_scans_share_the_plans_scratch(cuda):
    # No synchronisation between scans of different sizes on one plan: the
    # range sums of one are rewritten by the next.
    ranges = 5 * torch.cuda.get_device_properties(0).multi_processor_count
    sizes = [20_001, 7 * ranges * 4096 + 1, 4096 * 3, 2 * ranges * 4096 + 9, 50_000]
    xs = [_rand("u32", n, seed=n) for n in sizes]
    d_in = [_dev(x) for x in xs]
    outs = [torch.empty_like(d) for d in d_in]
    with Plan("rts", "u32", max_n=max(sizes)) as plan:
        plan.set_small_max(0)
        for _ in range(3):
            for d, o in zip(d_in, outs):
                plan.scan(d, out=o, inclusive=True)
        plan.check()
    for x, o in zip(xs, outs):
        assert np.array_equal(o.cpu().numpy().view(np.uint32), oracle.scan(x, True))


def test_replays_with_new_inputs(cuda):
    n = 3_000_001
    x = _rand("u32", n, seed=5)
    d, side = _dev(x), torch.cuda.Stream()
    out = torch.empty_like(d)
    with Plan("rts", "u32", max_n=n) as plan:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            with torch.cuda.graph(graph, stream=side):
                plan.scan(d, out=out, stream=side)
                plan.scan(out, out=out, stream=side)
        for k in range(3):
            y = np.roll(x, k)
            d.copy_(_dev(y))
            graph.replay()
            graph.replay()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy().view(np.uint32), oracle.scan(oracle.scan(y, False), False)), k
