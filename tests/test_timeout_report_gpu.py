"""gps_plan_check() reports a wait that ran past its budget on plans of every
element type, whether their kernels share one device header or have two."""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_forced_stalls(cuda, dtype):
    # Units withhold their aggregate for 5 ms, successors may wait 50 us.
    np_t, word = {"u32": (np.uint32, np.int32), "u64": (np.uint64, np.int64)}[dtype]
    n = 64 * 4096
    x = np.random.default_rng(7).integers(0, np.iinfo(np_t).max, size=n, dtype=np_t, endpoint=True)
    d = torch.from_numpy(x.view(word)).cuda()
    with Plan("csdl", dtype, max_n=n) as plan:
        plan.set_wait_budget(50_000)
        plan.set_stall(mode=1, period=4, seed=0, delay_ns=5_000_000, fallback_polls=0)
        plan.scan(d)
        assert plan.check_status() == _lib.GPS_ERR_TIMEOUT
        assert plan.check_status() == _lib.GPS_OK  # read and cleared
        plan.set_stall(mode=0)
        plan.set_wait_budget(1_000_000_000)
        out = plan.scan(d, inclusive=True)
        plan.check()
    assert np.array_equal(out.cpu().numpy().view(np_t), oracle.scan(x, True))


@pytest.mark.parametrize("dtype,members", [("u64", 1), ("f32", 1), ("f32c", 1), ("u32x4", 4)])
def test_a_batch_with_a_slow_tile(cuda, dtype, members):
    # Tile 3 ends with millions of empty segments, whose offsets it reads for
    # milliseconds; the tiles after it may wait 100 us.
    word, size = {"u64": (torch.int64, 8), "u32x4": (torch.int32, 16)}.get(dtype, (torch.float32, 4))
    tile = 16384 // size
    n = 20 * tile
    d = torch.ones(n * members, dtype=word, device="cuda")
    offs = torch.full((6_000_000,), 4 * tile - 1, dtype=torch.int32, device="cuda")
    offs[0], offs[-1] = 0, n
    with Plan("csdl", dtype, max_n=n) as plan:
        plan.set_wait_budget(100_000)
        plan.scan_segmented(d, offs)
        assert plan.check_status() == _lib.GPS_ERR_TIMEOUT
        assert plan.check_status() == _lib.GPS_OK
        plan.set_wait_budget(1_000_000_000)
        got = plan.scan_segmented(d, offs, inclusive=True).cpu().numpy().reshape(n, members)
        plan.check()
    want = np.concatenate([np.arange(1, 4 * tile), np.arange(1, n - 4 * tile + 2)])
    assert np.array_equal(got.astype(np.int64), np.repeat(want[:, None], members, axis=1))
