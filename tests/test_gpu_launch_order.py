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


def test_waits_count_from_the_end_of_the_kernel_before():
    """A kernel that is set up under one that runs for longer than the limit of its barrier waits (0.4 s): its waits begin when the
    other is done.  The long one is a plain-FMA product of one row and one column, one block for some tens of millions of terms."""
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(1)
    top = 1 << 27
    v = torch.rand(top, device=DEV, generator=g)
    dot = torch.empty(1, 1, device=DEV)
    small = capi.Gemm(False, True, 1, 1, 1 << 20, math_mode=capi.MATH_FP32_FFMA)

    def product(k):
        small.gemm(1, 1, k, v, k, v, k, dot, 1)

    def seconds(k):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        product(k)
        e[1].record()
        torch.cuda.synchronize()
        return e[0].elapsed_time(e[1]) * 1e-3

    seconds(1 << 16)
    terms = int((1 << 22) * 0.8 / seconds(1 << 22))
    assert terms <= top
    # one plan for each kernel with such waits: streamed matrix, staged 3x3, 1x1 over a large plane, general (7x7 planes)
    calls = []
    for make, x in [(lambda: capi.IPForward(2048, 1000, 8, bias=False), (8, 2048)),
                    (lambda: capi.Conv2DForward(channels_in=32, channels_out=64, kernel=3, pad=1, batch=2, height=56, width=56), (2, 32, 56, 56)),
                    (lambda: capi.Conv2DForward(channels_in=64, channels_out=64, kernel=1, batch=2, height=56, width=56), (2, 64, 56, 56)),
                    (lambda: capi.Conv2DForward(channels_in=64, channels_out=64, kernel=3, pad=1, batch=8, height=7, width=7), (8, 64, 7, 7))]:
        plan = make()
        w = (1000, 2048) if len(x) == 2 else (64, x[1], plan.desc.kernel[0], plan.desc.kernel[0])
        packed = plan.prepack(torch.randn(*w, device=DEV, generator=g))
        y = torch.full((8, 1000) if len(x) == 2 else (x[0], 64, x[2], x[3]), float("nan"), device=DEV)
        ws = torch.empty(max(plan.workspace(), 16), dtype=torch.uint8, device=DEV)
        calls.append((plan, torch.randn(*x, device=DEV, generator=g), packed, y, ws))
    for plan, x, packed, y, ws in calls:
        plan.enqueue_packed(x, packed, None, y, ws=ws)
        torch.cuda.synchronize()
        want = y.clone()
        y.fill_(float("nan"))
        torch.cuda.synchronize()
        start = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        start[0].record()
        product(terms)
        plan.enqueue_packed(x, packed, None, y, ws=ws)
        start[1].record()
        assert capi.device_status() == 0
        assert start[0].elapsed_time(start[1]) > 500
        assert torch.equal(y, want)
