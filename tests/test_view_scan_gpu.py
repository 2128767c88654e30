"""Large integer scans of views off a 16-byte boundary on the generic kernel: every
pair of element offsets, at the sizes where rows, tiles and units end, bit-exact
against a scan of aligned buffers that runs on the one-tile-per-CTA kernel, and
nothing written outside the output."""
import numpy as np
import pytest
import torch

import oracle
from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu

TORCH = {"u32": torch.int32, "u64": torch.int64}


@pytest.mark.parametrize("inclusive", [False, True])
@pytest.mark.parametrize("dtype", ["u32", "u64"])
def test_large_views_at_every_offset_pair(cuda, dtype, inclusive):
    es = 8 if dtype == "u64" else 4
    tile, row, offsets = 16384 // es, 128 // es, 16 // es
    # The kernel takes over at two units of 4 tiles per SM.
    first = 8 * torch.cuda.get_device_properties(0).multi_processor_count * tile
    sizes = [first + k for k in (0, 1, row - 1, row, tile - 3, tile - 1, tile, 4 * tile - 3, 4 * tile - 1, 4 * tile + 1,
                                 9 * tile + 3 * row + 2)]
    pad, top = 8, max(sizes)
    gen = torch.Generator(device="cuda").manual_seed(5)
    data = torch.randint(-(1 << 31), (1 << 31) - 1, (top + 4,), dtype=TORCH[dtype], device="cuda", generator=gen)
    x = torch.empty(top, dtype=TORCH[dtype], device="cuda")
    buf = torch.empty(top + offsets + 2 * pad, dtype=TORCH[dtype], device="cuda")
    with Plan("csdl", dtype, max_n=top) as plan, Plan("csdl", dtype, max_n=top) as mid:
        plan.set_mid_max(1)
        mid.set_mid_max(top)
        for i in range(offsets):
            x.copy_(data[i:i + top])  # aligned
            want = mid.scan(x, inclusive=inclusive)  # a prefix does not depend on n
            if i == 0:
                np_t = np.uint64 if dtype == "u64" else np.uint32
                ref = oracle.scan(x.cpu().numpy().view(np_t), inclusive)
                assert np.array_equal(want.cpu().numpy().view(np_t), ref)
            for n in sizes:
                for o in range(offsets):
                    buf.fill_(-7)
                    plan.scan(data[i:i + n], out=buf[pad + o:pad + o + n], inclusive=inclusive)
                    assert torch.equal(buf[pad + o:pad + o + n], want[:n]), (n, i, o)
                    assert bool((buf[:pad + o] == -7).all()) and bool((buf[pad + o + n:] == -7).all()), (n, i, o)
                work = data.clone()
                plan.scan(work[i:i + n], out=work[i:i + n], inclusive=inclusive)  # in place
                assert torch.equal(work[i:i + n], want[:n]), (n, i)
                assert torch.equal(work[:i], data[:i]) and torch.equal(work[i + n:], data[i + n:]), (n, i)
        plan.check()
        mid.check()
