"""A launch configuration read from one plan and set on another makes the same
launch there: the autotuner's choice, the untuned one, and one tile per CTA."""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan
from gpuprefixsums_gb300._lib import GpsError
from test_batched_gpu import dev, fp_input

pytestmark = pytest.mark.gpu


def _set(plan, n, cfg, segmented):
    plan.set_generic_config(n, cfg["unit_tiles"], cfg["ctas_div"], segmented=segmented,
                            threads_per_row=cfg["threads_per_row"])


@pytest.mark.parametrize("tuned", [False, True])
@pytest.mark.parametrize("n", [1 << 16, 1_000_003, 9_000_001])
def test_floating_point_scan(cuda, n, tuned):
    d = torch.from_numpy(fp_input("normal", n, seed=n)).cuda()
    with Plan("csdl", "f32", max_n=n) as a, Plan("csdl", "f32", max_n=n) as b:
        if tuned:
            choice = a.autotune(d)
            assert {k: a.generic_config(n, segmented=False)[k] for k in choice} == choice
        cfg = a.generic_config(n, segmented=False)
        assert cfg["tuned"] == tuned
        want = a.scan(d, inclusive=True)
        _set(b, n, cfg, False)
        assert b.generic_config(n, segmented=False) == {**cfg, "tuned": True}
        got = b.scan(d, inclusive=True)
        a.check()
        b.check()
        assert a.geometry(n)["grid"] == b.geometry(n)["grid"]
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))  # the same roundings


def test_one_tile_per_cta_where_the_untuned_choice_is_another(cuda):
    tile, n = 4096, 3000 * 4096 + 5
    rng = np.random.default_rng(1)
    x = rng.integers(0, 2 ** 32, size=n, dtype=np.uint64).astype(np.uint32)
    offs = np.array([0, 5, 2_000_000, n], dtype=np.uint64)
    d_off = torch.from_numpy(offs.astype(np.uint32).view(np.int32)).cuda()
    with Plan("csdl", "u32", max_n=4097 * tile) as plan:
        assert plan.generic_config(n)["unit_tiles"] == 4
        plan.set_generic_config(n, 0)
        assert plan.generic_config(n) == {"unit_tiles": 0, "ctas_div": 1, "threads_per_row": 1, "tuned": True}
        got = plan.scan_segmented(dev(x), d_off)
        assert plan.geometry(n)["grid"] == 3001
        assert np.array_equal(got.cpu().numpy().view(np.uint32), oracle.segscan(x, offs, False))
        # The kernel takes at most 4096 tiles, and the triple has one form.
        assert plan.generic_config(4097 * tile)["unit_tiles"] == 4
        for bad in ((4097 * tile, 0, 1, 1), (n, 0, 2, 1), (n, 0, 1, 2), (n, 2, 1, 1)):
            with pytest.raises(GpsError):
                plan.set_generic_config(bad[0], bad[1], bad[2], threads_per_row=bad[3])
        plan.check()
