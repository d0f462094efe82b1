"""Launches that may start under the kernel before them (one wave of blocks) and launches that may not: a chain of dependent calls
that nothing waits between gives, bit for bit, what the same calls give one at a time -- on a stream, and captured in a graph."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_util import DEV


@pytest.mark.parametrize("rows,captured", [(1, False), (1, True), (64, False), (64, True), (40000, False)])
def test_chain_of_dependent_launches(rows, captured):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(rows)
    n = 256
    w = [torch.randn(n, n, device=DEV, generator=g) * (2.0 / n) ** 0.5 for _ in range(2)]
    bias = torch.randn(n, device=DEV, generator=g) * 0.1
    x = torch.randn(rows, n, device=DEV, generator=g)
    plan = capi.IPForward(n, n, rows, bias=True, activation="relu")
    ws = torch.empty(max(plan.workspace(), 16), dtype=torch.uint8, device=DEV)        # shared: each call packs its weights over the last one's
    a, b = torch.empty_like(x), torch.empty_like(x)

    def chain(stream, wait):
        a.copy_(x)
        for i in range(12):
            plan.enqueue(a, w[i % 2], bias, b, ws=ws, stream=stream)
            wait()
            capi.elementwise(a, b, a, "sum", 0.5, 0.5, "relu", stream=stream)       # in place
            wait()
            capi.softmax(b, b, stream=stream)
            wait()
            capi.elementwise(a, b, a, "sum", 1.0, 1.0, "identity", stream=stream)
            wait()

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        chain(stream, stream.synchronize)
        want = a.clone()
        if captured:
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                chain(stream, lambda: None)
            for _ in range(3):
                graph.replay()
        else:
            for _ in range(3):
                chain(stream, lambda: None)
    torch.cuda.synchronize()
    assert capi.device_status() == 0
    assert torch.equal(a, want)
