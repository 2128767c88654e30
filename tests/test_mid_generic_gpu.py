"""Small and mid sizes of the batched, floating-point and struct scans (one
tile per CTA, mid_seg.cuh) against the oracle.

Sizes sit on the edges of the 16 KB tile, of the groups of 64 tiles the
lookback folds, and of the default size limits. Integer results are bit-exact. Floating-point
results are held to the bounds of the library's other scans: compensated FP32,
relative error <= 1e-6 (rounding the exact prefix to FP32 costs 2^-24) and
normwise <= 1e-7; plain FP32, normwise <= 1e-5; both repeat bit for bit.
"""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan
from test_batched_gpu import dev, fp_errors, fp_input, offsets_of

pytestmark = pytest.mark.gpu

NP = {"u32": np.uint32, "u64": np.uint64}


def _lengths(rng, n, style):
    """Segment lengths adding up to n: mostly short, or a few long ones, with empties."""
    if style == "short":
        cut = np.sort(rng.integers(0, n + 1, size=n // 2 + 600))  # many empty segments, several search rounds
    elif style == "long":
        cut = np.sort(rng.integers(0, n + 1, size=max(1, n // 50_000)))
    else:  # one segment, and empty ones at both ends
        cut = np.array([0, 0, n, n])
    return np.diff(np.concatenate([[0], cut, [n]]))


@pytest.mark.parametrize("style", ["short", "long", "one"])
@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_batched_integers(cuda, dtype, style):
    tile = 16384 // np.dtype(NP[dtype]).itemsize
    sizes = [1, 3, tile - 1, tile, tile + 1, 31 * tile + 7, 32 * tile, 32 * tile + 1, 33 * tile + 5, 64 * tile,
             65 * tile, 100 * tile + 9, 1216 * tile, 1217 * tile - 3, 1728 * tile, 2049 * tile - 1]
    with Plan("csdl", dtype, max_n=max(sizes)) as plan:
        for n in sizes:
            rng = np.random.default_rng(n)
            offs = offsets_of(_lengths(rng, n, style))
            x = rng.integers(0, np.iinfo(NP[dtype]).max, size=n, dtype=NP[dtype], endpoint=True)
            d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
            for inclusive in (False, True):
                d = dev(x)
                got = plan.scan_segmented(d, d_off, inclusive=inclusive)
                want = oracle.segscan(x, offs, inclusive)
                assert np.array_equal(got.cpu().numpy().view(NP[dtype]), want), (n, inclusive)
                plan.scan_segmented(d, d_off, out=d, inclusive=inclusive)  # in place
                assert np.array_equal(d.cpu().numpy().view(NP[dtype]), want), (n, inclusive)
        plan.check()


@pytest.mark.parametrize("inclusive", [False, True])
@pytest.mark.parametrize("dt", ["f32", "f32c"])
def test_floating_point(cuda, dt, inclusive):
    sizes = [1, 4095, 4097, 32 * 4096 + 1, 65 * 4096 - 2, 129 * 4096, 1216 * 4096 - 1, 1217 * 4096, 1281 * 4096 - 7,
             2049 * 4096 - 7]
    with Plan("csdl", dt, max_n=max(sizes)) as plan:
        for n in sizes:
            x = fp_input("mixed", n, seed=n)
            d = torch.from_numpy(x).cuda()
            got = plan.scan(d, inclusive=inclusive).cpu().numpy()
            again = plan.scan(d, inclusive=inclusive).cpu().numpy()
            assert np.array_equal(got.view(np.uint32), again.view(np.uint32)), n
            rel, _, norm = fp_errors(got, oracle.scan_f32_exact(x, inclusive=inclusive), x)
            if dt == "f32c":
                assert rel <= 1e-6 and norm <= 1e-7, (n, rel, norm)
            else:
                assert norm <= 1e-5, (n, norm)
        plan.check()


@pytest.mark.parametrize("dt", ["f32", "f32c"])
def test_an_infinity_stays_inside_its_segment(cuda, dt):
    # Segment 1 holds an infinity: the prefixes before it and the other
    # segments stay finite and right, whatever tile they are in.
    n, tile = 40 * 4096 + 17, 4096
    offs = np.array([0, 3 * tile + 5, 35 * tile + 9, n], dtype=np.uint64)
    x = fp_input("normal", n, seed=3)
    bad = 20 * tile + 100
    x[bad] = np.inf
    d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
    with Plan("csdl", dt, max_n=n) as plan:
        got = plan.scan_segmented(torch.from_numpy(x).cuda(), d_off, inclusive=True).cpu().numpy()
        plan.check()
    bound = 1e-7 if dt == "f32c" else 1e-5
    for b, e in ((0, int(offs[1])), (int(offs[1]), bad), (int(offs[2]), n)):
        assert fp_errors(got[b:e], oracle.scan_f32_exact(x[b:e], inclusive=True), x[b:e])[2] <= bound
    assert not np.any(np.isfinite(got[bad:int(offs[2])]))


@pytest.mark.parametrize("inclusive", [False, True])
def test_structs_plain_and_batched(cuda, inclusive):
    sizes = [1, 1023, 1025, 33 * 1024 + 1, 65 * 1024, 704 * 1024, 705 * 1024 + 3]
    with Plan("csdl", "u32x4", max_n=max(sizes)) as plan:
        for n in sizes:
            rng = np.random.default_rng(n)
            x = rng.integers(0, 2 ** 32, size=(n, 4), dtype=np.uint64).astype(np.uint32)
            d = dev(x.reshape(-1))
            got = plan.scan(d, inclusive=inclusive).cpu().numpy().view(np.uint32).reshape(n, 4)
            assert np.array_equal(got, oracle.scan_members(x, inclusive=inclusive)), n
            offs = offsets_of(_lengths(rng, n, "long" if n > 50_000 else "short"))
            d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
            got = plan.scan_segmented(d, d_off, inclusive=inclusive).cpu().numpy().view(np.uint32).reshape(n, 4)
            for m in range(4):
                want = oracle.segscan(np.ascontiguousarray(x[:, m]), offs, inclusive)
                assert np.array_equal(got[:, m], want), (n, m)
        plan.check()


def test_autotune_of_a_small_batch_keeps_results_and_reports_a_settable_configuration(cuda):
    rng = np.random.default_rng(9)
    n = 300_007
    offs = offsets_of(_lengths(rng, n, "long"))
    x = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
    want = oracle.segscan(x, offs, False)
    with Plan("csdl", "u32", max_n=n) as plan:
        choice = plan.autotune(dev(x), d_off)
        cfg = plan.generic_config(n)
        assert cfg["tuned"] and {k: cfg[k] for k in choice} == choice
        assert np.array_equal(plan.scan_segmented(dev(x), d_off).cpu().numpy().view(np.uint32), want)
        plan.set_generic_config(n, choice["unit_tiles"], choice["ctas_div"], threads_per_row=choice["threads_per_row"])
        assert np.array_equal(plan.scan_segmented(dev(x), d_off).cpu().numpy().view(np.uint32), want)
        plan.check()


def test_captured_batches_replay(cuda):
    # Replays of one captured launch get new grid ids: descriptors of the
    # replay before must not match.
    rng = np.random.default_rng(10)
    n = 200_003
    offs = offsets_of(_lengths(rng, n, "long"))
    d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
    x = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    d_x = dev(x)
    out = torch.empty_like(d_x)
    st = torch.cuda.Stream()
    with Plan("csdl", "u32", max_n=n) as plan:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.stream(st):
            with torch.cuda.graph(g, stream=st):
                plan.scan_segmented(d_x, d_off, out=out, stream=st)
        for k in range(3):
            y = np.roll(x, k)
            d_x.copy_(dev(y))
            g.replay()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy().view(np.uint32), oracle.segscan(y, offs, False)), k
        plan.check()


@pytest.mark.parametrize("count", [255, 1023, 1024, 1025, 2049, 70_000])
def test_segment_counts_around_one_reading(cuda, count):
    """A CTA reads up to 1024 offsets at once and narrows longer lists first."""
    n = 130 * 4096 + 11
    rng = np.random.default_rng(count)
    offs = np.concatenate([[0], np.sort(rng.integers(0, n + 1, size=count - 1)), [n]])
    x = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
    with Plan("csdl", "u32", max_n=n) as plan:
        for inclusive in (False, True):
            got = plan.scan_segmented(dev(x), d_off, inclusive=inclusive)
            assert np.array_equal(got.cpu().numpy().view(np.uint32), oracle.segscan(x, offs, inclusive))
        plan.check()
