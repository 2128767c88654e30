"""Waits of the one-tile-per-CTA kernels that run past the plan's budget.

One tile of a batch is kept busy for milliseconds by millions of empty segments
at its end, whose offsets it has to read; with a budget of 100 us the tiles
after it give up, and the launch number stays behind with descriptors under it.
Until the timeout has been reported, later calls may leave their outputs
undefined, but write nothing outside them, and a select, whose output position
is what it would wait for, writes nothing at all. Once it has been reported,
every call on the plan is exact again.
"""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan, _lib, lib

pytestmark = pytest.mark.gpu

NP = {"u32": np.uint32, "u64": np.uint64, "f32": np.float32}
WORD = {"u32": np.int32, "u64": np.int64, "f32": np.float32}
TILE_BYTES = 16384


def _dev(dtype, x):
    return torch.from_numpy(np.ascontiguousarray(x).view(WORD[dtype])).cuda()


def _exact(plan, dtype, x, d, d_off, offs, flags):
    """Scans, batches and selects on the plan, twice: both sets of group sums."""
    for _ in range(2):
        got = plan.scan_segmented(d, d_off, inclusive=True).cpu().numpy().view(NP[dtype])
        sel, count = plan.select(d, torch.from_numpy(flags).cuda())
        assert int(count.item()) == int(flags.sum())
        assert np.array_equal(sel.cpu().numpy().view(NP[dtype])[:int(flags.sum())], x[flags != 0])
        full = plan.scan(d, inclusive=True).cpu().numpy().view(NP[dtype])
        if dtype == "f32":  # small whole numbers: every partial sum is exact
            assert np.array_equal(full, np.cumsum(x, dtype=np.float64).astype(np.float32))
            want = np.concatenate([np.cumsum(x[b:e], dtype=np.float64) for b, e in zip(offs, offs[1:])])
            assert np.array_equal(got, want.astype(np.float32))
        else:
            assert np.array_equal(full, oracle.scan(x, True))
            assert np.array_equal(got, oracle.segscan(x, offs, True))
    plan.check()


@pytest.mark.parametrize("tiles", [20, 300])  # one group of tiles; several
@pytest.mark.parametrize("dtype", ["u32", "u64", "f32"])
def test_an_expired_wait_is_reported_and_leaves_the_plan_usable(cuda, dtype, tiles):
    tile = TILE_BYTES // np.dtype(NP[dtype]).itemsize
    n = tiles * tile - 7
    rng = np.random.default_rng(tiles)
    top = 16 if dtype == "f32" else np.iinfo(NP[dtype]).max
    x = rng.integers(0, top, size=n, dtype=np.uint64 if dtype != "u32" else np.uint32).astype(NP[dtype])
    flags = (rng.random(n) < 0.4).astype(np.uint8)
    d, d_flags = _dev(dtype, x), torch.from_numpy(flags).cuda()
    offs = np.unique(np.concatenate([[0, n], rng.integers(0, n, size=30)])).astype(np.uint64)
    d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
    slow = torch.full((6_000_000,), 4 * tile - 1, dtype=torch.int32, device="cuda")
    slow[0], slow[-1] = 0, n
    count = torch.full((1,), -5, dtype=torch.int64, device="cuda")
    sel = torch.full((n + 16,), -3, dtype=d.dtype, device="cuda")
    out = torch.full((n + 16,), -3, dtype=d.dtype, device="cuda")
    with Plan("csdl", dtype, max_n=n) as plan:
        _exact(plan, dtype, x, d, d_off, offs, flags)
        for budget_reset_first in (False, True):
            plan.set_wait_budget(100_000)
            plan.scan_segmented(d, slow, out=out[:n])
            if budget_reset_first:
                plan.set_wait_budget(1_000_000_000)
            # Not reported yet: the next launches find the flag.
            plan.select(d, d_flags, out=sel[8:8 + n], num_selected=count)
            plan.scan(d, out=out[:n])
            plan.scan_segmented(d, d_off, out=out[:n])
            plan.select(d, d_flags, out=sel[8:8 + n], num_selected=count)
            assert plan.check_status() == _lib.GPS_ERR_TIMEOUT
            assert int(count.item()) == -5 and bool((sel == -3).all())
            assert bool((out[n:] == -3).all())
            assert plan.check_status() == _lib.GPS_OK
            plan.set_wait_budget(1_000_000_000)
            _exact(plan, dtype, x, d, d_off, offs, flags)


@pytest.mark.parametrize("op", ["scan", "select"])
def test_a_wait_on_slow_loads(cuda, op):
    # Values in pinned host memory arrive at one tile tens of microseconds
    # after another; a wait may take 17 polls at most (a budget of 1 ns).
    n = 3_000_001
    rng = np.random.default_rng(11)
    x = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    flags = (rng.random(n) < 0.4).astype(np.uint8)
    offs = np.array([0, 70_001, n], dtype=np.uint64)
    d, d_flags = _dev("u32", x), torch.from_numpy(flags).cuda()
    d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
    h = torch.from_numpy(x.view(np.int32)).pin_memory()
    out = torch.empty_like(d)
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    with Plan("csdl", "u32", max_n=n) as plan:
        for _ in range(2):
            plan.set_wait_budget(1)
            for _ in range(50):
                if op == "scan":
                    plan.scan_ptr(h.data_ptr(), out.data_ptr(), n)
                else:
                    assert lib.gps_select_flagged(plan.handle, h.data_ptr(), d_flags.data_ptr(), out.data_ptr(), n,
                                                  count.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
                status = plan.check_status()
                if status != _lib.GPS_OK:
                    break
            assert status == _lib.GPS_ERR_TIMEOUT
            plan.set_wait_budget(1_000_000_000)
            _exact(plan, "u32", x, d, d_off, offs, flags)
