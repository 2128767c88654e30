"""Integer scans of views at every element offset from a 16-byte boundary, on
both sides, against the oracle: bit-exact, nothing written outside the
output. The one-tile-per-CTA kernel counts its tiles from the boundary below
the input, so the edges lie `offset` elements before the tile sizes."""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu

NP = {"u32": np.uint32, "u64": np.uint64}
SIGNED = {"u32": np.int32, "u64": np.int64}


def _rand(dtype, n, seed):
    return np.random.default_rng(seed).integers(0, np.iinfo(NP[dtype]).max, size=n, dtype=NP[dtype], endpoint=True)


@pytest.mark.parametrize("inclusive", [False, True])
@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_views_at_every_offset_pair(cuda, dtype, inclusive):
    tile = 16384 // np.dtype(NP[dtype]).itemsize
    offsets = range(4) if dtype == "u32" else range(2)
    sizes = [1, 2, 3, 5, tile - 3, tile - 1, tile, tile + 1, 2 * tile + 2, 32 * tile - 1, 32 * tile + 1, 33 * tile]
    pad = 8
    with Plan("csdl", dtype, max_n=max(sizes)) as plan:
        for n in sizes:
            x = _rand(dtype, n, seed=n)
            want = oracle.scan(x, inclusive)
            for i in offsets:
                src = torch.from_numpy(np.concatenate([_rand(dtype, i, 1), x]).view(SIGNED[dtype])).cuda()
                for o in offsets:
                    buf = torch.full((pad + o + n + pad,), -7, dtype=src.dtype, device="cuda")
                    plan.scan(src[i:], out=buf[pad + o:pad + o + n], inclusive=inclusive)
                    got = buf.cpu().numpy()
                    assert np.array_equal(got[pad + o:pad + o + n].view(NP[dtype]), want), (n, i, o)
                    assert np.all(got[:pad + o] == -7) and np.all(got[pad + o + n:] == -7), (n, i, o)
                plan.scan(src[i:], out=src[i:], inclusive=inclusive)  # in place
                assert np.array_equal(src[i:].cpu().numpy().view(NP[dtype]), want), (n, i)
        plan.check()


@pytest.mark.parametrize("in_off,out_off", [(1, 0), (0, 3), (2, 2)])
def test_a_large_view_above_the_mid_size(cuda, in_off, out_off):
    n = (1 << 24) + 3 * 4096 + 5  # past 64 MB, where aligned buffers take the persistent kernel
    x = _rand("u32", n, seed=24)
    src = torch.empty(n + in_off, dtype=torch.int32, device="cuda")
    src[in_off:] = torch.from_numpy(x.view(np.int32)).cuda()
    out = torch.empty(n + out_off, dtype=torch.int32, device="cuda")
    with Plan("csdl", "u32", max_n=n) as plan:
        plan.scan(src[in_off:], out=out[out_off:])
        plan.check()
    assert oracle.validate(x, out[out_off:].cpu().numpy().view(np.uint32), False) == 0
