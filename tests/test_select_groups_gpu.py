"""Stream compaction around the edges of the persistent kernel's split: units of
4 tiles, whose tiles go to two groups of finalize warps in turn, on plans
whose launches end in the middle of a unit. Bit-exact against the oracle,
nothing written past the count."""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu

NP = {"u32": np.uint32, "u64": np.uint64}
SIGNED = {"u32": np.int32, "u64": np.int64}


@pytest.mark.parametrize("density", [0.0, 0.03, 0.5, 1.0])
@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_units_and_groups(cuda, dtype, density):
    tile = 16384 // np.dtype(NP[dtype]).itemsize
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    big = 4 * tile * (sms * 10)  # more units per CTA than are in flight
    sizes = [big, big + tile, big + 2 * tile - 5, big + 3 * tile + 1, big - 4 * tile + 17]
    rng = np.random.default_rng(int(density * 100))
    x = rng.integers(0, np.iinfo(NP[dtype]).max, size=max(sizes), dtype=NP[dtype], endpoint=True)
    fl = (rng.random(max(sizes)) < density).astype(np.uint8) * 3
    d, d_fl = torch.from_numpy(x.view(SIGNED[dtype])).cuda(), torch.from_numpy(fl).cuda()
    with Plan("csdl", dtype, max_n=max(sizes)) as plan:
        for shift, n in enumerate(sizes):
            want = oracle.select(x[:n], fl[:n])
            out = torch.full((n + 8,), -1, dtype=d.dtype, device="cuda")
            _, cnt = plan.select(d[:n], d_fl[:n], out=out[shift:])  # every phase of the output
            got = out.cpu().numpy()
            assert int(cnt.item()) == want.size
            assert np.array_equal(got[shift:shift + want.size].view(NP[dtype]), want)
            assert np.all(got[:shift] == -1) and np.all(got[shift + want.size:] == -1)
        plan.check()
