"""Buffers at addresses that 16-byte accesses cannot take: scratch that starts off a boundary (the same parts, the same bits), and
matrices of a batch at strides that are no multiple of four."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_util import DEV


@pytest.mark.parametrize("shift", [4, 8, 12])
def test_scratch_at_any_address(shift):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(shift)
    ip = capi.IPForward(2048, 1000, 5, bias=True, activation="relu")
    conv = capi.Conv2DForward(channels_in=512, channels_out=512, kernel=3, pad=1, batch=1, height=7, width=7, bias=True)
    for plan, x, w, shape in [(ip, (5, 2048), (1000, 2048), (5, 1000)), (conv, (1, 512, 7, 7), (512, 512, 3, 3), (1, 512, 7, 7))]:
        xt = torch.randn(*x, device=DEV, generator=g)
        packed = plan.prepack(torch.randn(*w, device=DEV, generator=g))
        bias = torch.randn(w[0], device=DEV, generator=g)
        ws = torch.empty(plan.workspace() + shift, dtype=torch.uint8, device=DEV)
        y, y2 = (torch.full(shape, float("nan"), device=DEV) for _ in range(2))
        plan.enqueue_packed(xt, packed, bias, y, ws=ws)
        plan.enqueue_packed(xt, packed, bias, y2, ws=ws[shift:])
        assert capi.device_status() == 0
        assert bool(y.isfinite().all()) and torch.equal(y, y2)


@pytest.mark.parametrize("extra", [1, 2, 3, 4])
def test_batched_matrices_at_any_stride(extra):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(extra)
    count, m, n, k = 3, 130, 96, 64
    stride = m * k + extra
    a = torch.randn(count * stride, device=DEV, generator=g)
    b = torch.randn(count, n, k, device=DEV, generator=g)
    plan = capi.Gemm(False, True, m, n, k)
    c = torch.full((count, m, n), float("nan"), device=DEV)
    ws = torch.empty(plan.batched_workspace(count), dtype=torch.uint8, device=DEV)
    plan.batch_gemm(count, m, n, k, a, stride, k, b, n * k, k, c, m * n, n, ws=ws)
    assert capi.device_status() == 0
    rows = torch.stack([a[i * stride:i * stride + m * k].view(m, k) for i in range(count)])
    want = torch.matmul(rows.double(), b.double().transpose(1, 2))
    assert float((c.double() - want).norm() / want.norm()) < 5e-6       # as in test_gpu_stream.py
