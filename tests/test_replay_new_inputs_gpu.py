"""Replays of captured scans whose inputs change between replays.

A replay must not take a descriptor of an earlier replay for its own: the
launch's tag may not be one that is fixed when the graph is instantiated.
Each captured graph holds the only scans of its plan, so the descriptors a
replay finds are those of the replay before.
"""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu


def _dev(x):
    return torch.from_numpy(x.view({4: np.int32, 8: np.int64}[x.itemsize])).cuda()


@pytest.mark.parametrize("sizes", [(200_003,), (33 * 4096, 5 * 4096 + 1), (1 << 21, 70_001, 4097)])
@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_replays_with_new_inputs(cuda, dtype, sizes):
    np_t = {"u32": np.uint32, "u64": np.uint64}[dtype]
    rng = np.random.default_rng(sum(sizes))
    xs = [rng.integers(0, np.iinfo(np_t).max, size=n, dtype=np_t, endpoint=True) for n in sizes]
    d_in = [_dev(x) for x in xs]
    outs = [torch.empty_like(d) for d in d_in]
    side = torch.cuda.Stream()
    with Plan("csdl", dtype, max_n=max(sizes)) as plan:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            with torch.cuda.graph(graph, stream=side):
                for d, o in zip(d_in, outs):
                    plan.scan(d, out=o, stream=side)
        for k in range(4):
            ys = [np.roll(x, 7 * k) for x in xs]
            for d, y in zip(d_in, ys):
                d.copy_(_dev(y))
            graph.replay()
            torch.cuda.synchronize()
            for o, y in zip(outs, ys):
                assert np.array_equal(o.cpu().numpy().view(np_t), oracle.scan(y, False)), (k, y.size)
            if k == 1:  # an eager scan between replays
                eager = plan.scan(d_in[0], inclusive=True)
                assert np.array_equal(eager.cpu().numpy().view(np_t), oracle.scan(ys[0], True))
        plan.check()
