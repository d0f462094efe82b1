"""The contraction kernel whose A operand the copy engines bring in (csrc/stream_tc.cu), at the sizes where its tiles, units and
slots end: rows around multiples of 128, images that end inside a tile, K around multiples of 32 and of the chunk of 256, ragged
columns, each column tile, split K -- against the same product in 64 bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_util import DEV

# 3xTF32: a product term is off by at most 2^-21 of itself (two operands, each carried to 22 bits), the sums of eight k-blocks
# inside the tensor core truncate at 2^-23 of the largest partial sum per step: 96 steps, 1.1e-5 in the worst case and a fraction
# of that for data of both signs.  Measured 2.2e-6 (2-norm); the bound is 5e-6.
TOL = 5e-6


def err(got, want):
    return float((got.double() - want).norm() / want.norm())


def off_boundary(t):
    """The same values four bytes off a 16-byte boundary, where no tensor map can start: the general kernel's problem."""
    return torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)


@pytest.mark.parametrize("ta,tb,m,n,k", [
    (False, True, 128, 128, 256), (False, True, 129, 128, 32), (False, True, 127, 130, 260), (False, True, 1, 1000, 2048),
    (False, False, 300, 33, 68), (False, True, 257, 64, 1024), (False, True, 2048, 96, 292), (False, True, 640, 32, 36),
    (True, False, 128, 128, 64), (True, False, 132, 200, 33), (True, True, 516, 65, 300), (True, False, 4, 20, 4100), (True, True, 1028, 31, 257),
])
def test_gemm(ta, tb, m, n, k):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(m * 7 + n)
    a = torch.randn(*((k, m) if ta else (m, k)), device=DEV, generator=g)
    b = torch.randn(*((n, k) if tb else (k, n)), device=DEV, generator=g)
    bias = torch.randn(n, device=DEV, generator=g)
    plan = capi.Gemm(ta, tb, m, n, k, bias_mode=2, activation="relu")
    c = torch.full((m, n), float("nan"), device=DEV)
    ws = torch.empty(max(plan.workspace(), 16), dtype=torch.uint8, device=DEV)
    plan.gemm(m, n, k, a, m if ta else k, b, k if tb else n, c, n, bias=bias, ws=ws)
    assert capi.device_status() == 0
    kernel, bn, parts = capi.last_route()
    assert kernel == ("stream_units" if ta else "stream_k") and bn == (32 if n <= 32 else 64 if n <= 64 else 128)
    want = torch.relu((a.double().t() if ta else a.double()) @ (b.double().t() if tb else b.double()) + bias.double())
    assert err(c, want) < TOL
    # the general kernel's bits
    c2 = torch.full((m, n), float("nan"), device=DEV)
    plan.gemm(m, n, k, off_boundary(a), m if ta else k, b, k if tb else n, c2, n, bias=bias, ws=ws)
    assert capi.device_status() == 0 and capi.last_route() == ("general_strided", bn, parts)
    assert torch.equal(c, c2)


@pytest.mark.parametrize("count,ta,m,n,k", [(5, False, 200, 150, 128), (16, True, 132, 256, 96), (3, False, 64, 33, 512)])
def test_batched_gemm(count, ta, m, n, k):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(count)
    a = torch.randn(count, *((k, m) if ta else (m, k)), device=DEV, generator=g)
    b = torch.randn(count, n, k, device=DEV, generator=g)
    plan = capi.Gemm(ta, True, m, n, k)
    c = torch.full((count, m, n), float("nan"), device=DEV)
    ws = torch.empty(max(plan.batched_workspace(count), 16), dtype=torch.uint8, device=DEV)
    plan.batch_gemm(count, m, n, k, a, m * k, m if ta else k, b, n * k, k, c, m * n, n, ws=ws)
    assert capi.device_status() == 0 and capi.last_route()[0] == ("stream_units" if ta else "stream_k")
    want = torch.matmul(a.double().transpose(1, 2) if ta else a.double(), b.double().transpose(1, 2))
    assert err(c, want) < TOL


# planes: pitches that the copy engines cannot take (7x7, 9x9, 27x27: the copying warp, from 16 taps on); one that ends inside a tile (14x14, 28x28), several per tile (8x8, 6x6: 36 pixels), one tile and a bit (12x12), wide rows
# kernel: the route of a launch that does not cut K.  One that does stays on it when a part is whole blocks of channels.
@pytest.mark.parametrize("batch,cin,cout,h,w,k,dil,kernel", [
    (1, 64, 128, 7, 7, 3, 1, "general_taps"), (9, 96, 130, 7, 7, 5, 1, "stream_copy"), (2, 64, 192, 27, 27, 5, 1, "stream_copy"),
    (5, 32, 64, 9, 9, 5, 1, "stream_copy"), (3, 64, 33, 5, 13, 5, 1, "stream_copy"), (2, 64, 128, 14, 14, 3, 1, "stream_units"),
    (5, 96, 160, 14, 14, 3, 1, "stream_units"), (3, 64, 128, 28, 28, 3, 1, "stream_units"), (2, 32, 192, 28, 28, 5, 1, "stream_units"),
    (4, 64, 128, 12, 12, 3, 2, "stream_units"), (6, 64, 100, 8, 8, 3, 1, "stream_units"), (13, 32, 128, 6, 6, 3, 1, "stream_units"),
    (1, 128, 128, 56, 56, 3, 1, "stream_units"), (2, 64, 64, 10, 20, 3, 1, "staged"), (3, 512, 512, 14, 14, 3, 1, "stream_units"),
])
def test_convolution(batch, cin, cout, h, w, k, dil, kernel):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(cin + cout + h)
    x = torch.randn(batch, cin, h, w, device=DEV, generator=g)
    wt = torch.randn(cout, cin, k, k, device=DEV, generator=g) * (2.0 / (cin * k * k)) ** 0.5
    bias = torch.randn(cout, device=DEV, generator=g)
    pad = dil * (k - 1) // 2
    plan = capi.Conv2DForward(channels_in=cin, channels_out=cout, kernel=k, pad=pad, dilate=dil, batch=batch, height=h, width=w, bias=True,
                              activation="relu")
    res = torch.randn(batch, cout, h, w, device=DEV, generator=g)
    packed = plan.prepack(wt)
    cols = torch.nn.functional.unfold(x.double(), (k, k), dilation=dil, padding=pad)
    want = torch.relu(torch.matmul(wt.double().reshape(cout, -1), cols).reshape(batch, cout, h, w) + bias.double()[None, :, None, None])
    for ws in (torch.empty(max(plan.workspace(), 16), dtype=torch.uint8, device=DEV), None):
        y, y2, y3 = (torch.full_like(res, float("nan")) for _ in range(3))
        plan.enqueue_packed(x, packed, bias, y, ws=ws)
        route = capi.last_route()
        if ws is None:
            assert route[0] == kernel and route[2] == 1
        elif kernel.startswith("stream") and (cin // 32) % route[2] == 0:
            assert route[0] == kernel
        plan.enqueue_packed(x, packed, bias, y2, residual=res, post_activation="relu6", ws=ws)
        assert capi.device_status() == 0
        assert err(y, want) < TOL
        assert err(y2, (want + res.double()).clamp(0, 6)) < TOL
        # units against the general kernel, or with many taps against the copying warp: the same bits
        plan.enqueue_packed(off_boundary(x), packed, bias, y3, ws=ws)
        assert capi.device_status() == 0
        if route[0] == "stream_units":
            assert capi.last_route() == ("general_taps" if k * k < 16 else "stream_copy", *route[1:])
            assert torch.equal(y, y3)
        else:
            assert err(y3, want) < TOL
