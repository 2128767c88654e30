"""Plan.geometry()'s launch count: that of the last scan, where it had as many
elements, else that of a scan of aligned buffers. A view off a 16-byte boundary may
count one tile more, and a mid-size scan of more than 4096 tiles runs in pieces.
Counted against the kernel nodes of the same call, captured."""
import ctypes

import pytest
import torch

from gpuprefixsums_gb300 import Plan

pytestmark = pytest.mark.gpu


def _nodes(plan, src, out):
    rt = ctypes.CDLL("libcudart.so.13")
    side = torch.cuda.Stream()
    handle = ctypes.c_void_p(side.cuda_stream)
    graph, count = ctypes.c_void_p(), ctypes.c_size_t()
    assert rt.cudaStreamBeginCapture(handle, 2) == 0  # relaxed
    plan.scan(src, out=out, stream=side)
    assert rt.cudaStreamEndCapture(handle, ctypes.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(count)) == 0
    assert rt.cudaGraphDestroy(graph) == 0
    return count.value


@pytest.mark.parametrize("off", [0, 1])
def test_reduce_then_scan(cuda, off):
    n = 2 * 5 * torch.cuda.get_device_properties(0).multi_processor_count * 4096  # whole chunks exactly
    x = torch.ones(n + off, dtype=torch.int32, device="cuda")[off:]
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    with Plan("rts", "u32", max_n=n) as plan:
        assert plan.geometry(n)["launches"] == 2  # nothing scanned yet
        plan.scan(x, out=out)
        assert plan.geometry(n)["launches"] == 2 + off == _nodes(plan, x, out)
        plan.scan(x, out=out, n=5000)
        assert plan.geometry(5000)["launches"] == 1  # one CTA
        assert plan.geometry(n)["launches"] == 2
        assert plan.geometry(n + 1)["launches"] == 3
        assert plan.geometry(0)["launches"] == 0
        plan.check()


@pytest.mark.parametrize("off", [0, 1])
def test_mid_size_scans_in_pieces(cuda, off):
    n = 4096 * 4096
    x = torch.ones(n + 1 + off, dtype=torch.int32, device="cuda")[off:]
    out = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    with Plan("csdl", "u32", max_n=n + 1) as plan:
        assert plan.geometry(n)["launches"] == 1 and plan.geometry(n + 1)["launches"] == 1
        plan.set_mid_max(n + 1)
        assert plan.geometry(n)["launches"] == 1 and plan.geometry(n + 1)["launches"] == 2
        plan.scan(x[:n], out=out[:n])
        assert plan.geometry(n)["launches"] == 1 + off == _nodes(plan, x[:n], out[:n])
        plan.scan(x, out=out)
        assert plan.geometry(n + 1)["launches"] == 2 == _nodes(plan, x, out)
        plan.set_mid_max(0)
        assert plan.geometry(n + 1)["launches"] == 1
        plan.check()
        assert bool((out.long() == torch.arange(n + 1, device="cuda")).all())
