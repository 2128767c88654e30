"""Plain integer chained scans on both sides of every size at which the kernel
changes (one tile per CTA, generic kernel, L2 kernel), aligned buffers, out of
place and in place, exclusive and inclusive: bit-exact against the oracle,
nothing written past the end."""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu

NP = {"u32": np.uint32, "u64": np.uint64}
SIGNED = {"u32": np.int32, "u64": np.int64}


def _check(plan, dtype, n, inclusive):
    x = np.random.default_rng(n).integers(0, np.iinfo(NP[dtype]).max, size=n, dtype=NP[dtype], endpoint=True)
    want = oracle.scan(x, inclusive)
    d = torch.from_numpy(x.view(SIGNED[dtype])).cuda()
    out = torch.full((n + 4,), -5, dtype=d.dtype, device="cuda")
    plan.scan(d, out=out, inclusive=inclusive)
    got = out.cpu().numpy()
    assert np.array_equal(got[:n].view(NP[dtype]), want) and np.all(got[n:] == -5), n
    plan.scan(d, out=d, inclusive=inclusive)
    assert np.array_equal(d.cpu().numpy().view(NP[dtype]), want), n


@pytest.mark.parametrize("inclusive", [False, True])
@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_sizes_where_the_kernel_changes(cuda, dtype, inclusive):
    es = np.dtype(NP[dtype]).itemsize
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    mid = (153 << 18) // es
    units = 8 * sms * 16384 // es  # with mid_max 0: fewest tiles the generic kernel takes
    with Plan("csdl", dtype, max_n=mid + 4096) as plan:
        for n in (mid - 1, mid, mid + 1, mid + 4096):
            _check(plan, dtype, n, inclusive)
        plan.set_mid_max(0)
        for n in (units - 16384 // es, units - 16384 // es + 1, units + 3):
            _check(plan, dtype, n, inclusive)
        plan.check()


def test_u32_beyond_512_mb(cuda):
    n = 1 << 27
    with Plan("csdl", "u32", max_n=n + 33) as plan:
        _check(plan, "u32", n, False)
        _check(plan, "u32", n + 33, True)
        plan.check()
