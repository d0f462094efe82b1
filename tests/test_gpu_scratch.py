"""Calls with packed weights whose scratch starts four bytes off a 16-byte boundary: the same parts, the same bits."""
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
