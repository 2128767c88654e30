"""The one-tile-per-CTA integer scans on one plan, in sequences whose launches use the
two sets of group sums in turn: sizes at the edges of groups of 32 tiles and of the
4096 tiles of a launch (more run in pieces), with scans that use no group sums,
batches and selects in between. Bit-exact against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu

NP = {"u32": np.uint32, "u64": np.uint64}
SIGNED = {"u32": np.int32, "u64": np.int64}


@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_sequences_of_sizes(cuda, dtype, off):
    tile = 16384 // np.dtype(NP[dtype]).itemsize
    tiles = [33, 33, 1, 64, 32, 65, 4096, 2, 1024, 1025, 40, 4097, 96, 8193, 34]
    top = max(tiles) * tile + 7
    # All bits in use: halves of u64 values carry into each other.
    x = np.random.default_rng(3).integers(0, np.iinfo(NP[dtype]).max, size=top, dtype=NP[dtype], endpoint=True)
    want = {inc: torch.from_numpy(oracle.scan(x, inc).view(SIGNED[dtype])).cuda() for inc in (False, True)}
    d = torch.empty(top + off, dtype=want[True].dtype, device="cuda")[off:]
    d.copy_(torch.from_numpy(x.view(SIGNED[dtype])))
    flags = torch.ones(50 * tile, dtype=torch.uint8, device="cuda")
    with Plan("csdl", dtype, max_n=top) as plan:
        plan.set_mid_max(top)
        for k, t in enumerate(tiles):
            for n in (t * tile - 1, t * tile, t * tile + 5):
                inc = bool((k + n) & 1)
                out = torch.full((n + 1,), -5, dtype=d.dtype, device="cuda")
                plan.scan(d[:n], out=out[:n], inclusive=inc)
                assert torch.equal(out[:n], want[inc][:n]) and int(out[n]) == -5, (t, n, inc)
            if off == 0 and k % 3 == 0:
                got, count = plan.select(d[:50 * tile], flags)[:2]
                assert int(count) == 50 * tile and torch.equal(got[:50 * tile], d[:50 * tile])
        plan.check()
