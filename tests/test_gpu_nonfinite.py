"""NaN and infinity through the dense kernels: a NaN comes out where the plain-FMA kernel has one (through the identity it stays, relu
and relu6 make it 0), and nowhere else; an infinity reaches the same outputs as something that is not finite (its TF32 remainder is
inf - inf, so it arrives as a NaN)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_util import DEV

BAD = [float("nan"), float("inf"), float("-inf")]


def check(call, act, value):
    """call(math mode) -> result"""
    from dlprimitives_b200 import capi
    got, want = call(capi.MATH_AUTO), call(capi.MATH_FP32_FFMA)
    assert capi.device_status() == 0
    if value != value:
        assert torch.equal(got.isnan(), want.isnan()) and (act != "identity" or bool(want.isnan().any()))
    else:
        assert torch.equal(got.isfinite(), want.isfinite()) and not bool(want.isfinite().all())
    assert torch.allclose(got[want.isfinite()], want[want.isfinite()], rtol=1e-4, atol=1e-4)


# (rows, outputs): full and partial column tiles of each width; K cut in parts and, without scratch, not
@pytest.mark.parametrize("rows,inputs,outputs", [(5, 2048, 1000), (130, 512, 128), (64, 512, 10), (300, 260, 64), (40, 1001, 200)])
@pytest.mark.parametrize("scratch", [True, False])
@pytest.mark.parametrize("act,value", [("identity", v) for v in BAD] + [("relu", BAD[0]), ("relu6", BAD[0])])
def test_inner_product(rows, inputs, outputs, scratch, act, value):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(rows)
    x, w, bias = torch.randn(rows, inputs, device=DEV, generator=g), torch.randn(outputs, inputs, device=DEV, generator=g) / inputs ** 0.5, torch.randn(outputs, device=DEV, generator=g)
    x[rows // 2, inputs // 3] = value
    x[rows - 1, 0] = value
    if value != value:
        w[outputs - 1, 5] = value

    def call(mode):
        plan = capi.IPForward(inputs, outputs, rows, bias=True, activation=act, math_mode=mode)
        y = torch.zeros(rows, outputs, device=DEV)
        ws = torch.empty(max(plan.workspace(), 16), dtype=torch.uint8, device=DEV) if scratch else None
        plan.enqueue_packed(x, plan.prepack(w), bias, y, ws=ws)
        return y
    check(call, act, value)


# staged; streamed, by units and by copies; general (7x7, stride 2, few channels); 1x1 over large planes and over small ones
@pytest.mark.parametrize("cin,cout,hw,k,stride", [(64, 64, 56, 3, 1), (64, 128, 28, 3, 1), (64, 192, 27, 5, 1), (64, 130, 7, 3, 1), (128, 64, 28, 3, 2), (3, 64, 32, 7, 2),
                                                  (20, 33, 15, 3, 1), (64, 64, 56, 1, 1), (256, 40, 28, 1, 1), (512, 128, 14, 1, 1)])
@pytest.mark.parametrize("act,value", [("identity", v) for v in BAD] + [("relu", BAD[0]), ("relu6", BAD[0])])
def test_convolution(cin, cout, hw, k, stride, act, value):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(hw)
    x, w, bias = torch.randn(3, cin, hw, hw, device=DEV, generator=g), torch.randn(cout, cin, k, k, device=DEV, generator=g) / (cin * k * k) ** 0.5, torch.randn(cout, device=DEV, generator=g)
    x[1, cin // 2, hw // 2, 2] = value
    x[2, 0, hw - 1, hw - 1] = value

    def call(mode):
        plan = capi.Conv2DForward(channels_in=cin, channels_out=cout, kernel=k, pad=k // 2, stride=stride, batch=3, height=hw, width=hw, bias=True, activation=act,
                                  math_mode=mode)
        y = torch.zeros(plan.output_shape(3), device=DEV)
        plan.enqueue(x, w, bias, y, ws=torch.empty(max(plan.workspace(), 16), dtype=torch.uint8, device=DEV))
        return y
    check(call, act, value)


# a NaN in the residual, through the activation after the sum
@pytest.mark.parametrize("cin,cout,hw,k", [(64, 128, 28, 3), (64, 64, 56, 1), (512, 128, 14, 1), (64, 130, 7, 3)])
@pytest.mark.parametrize("act", ["identity", "relu"])
def test_residual(cin, cout, hw, k, act):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(hw)
    x, w = torch.randn(3, cin, hw, hw, device=DEV, generator=g), torch.randn(cout, cin, k, k, device=DEV, generator=g) / (cin * k * k) ** 0.5
    res = torch.randn(3, cout, hw, hw, device=DEV, generator=g)
    res[1, cout // 2, 3, 3] = float("nan")

    def call(mode):
        plan = capi.Conv2DForward(channels_in=cin, channels_out=cout, kernel=k, pad=k // 2, batch=3, height=hw, width=hw, math_mode=mode)
        y = torch.zeros(3, cout, hw, hw, device=DEV)
        plan.enqueue_packed(x, plan.prepack(w), None, y, residual=res, post_activation=act,
                            ws=torch.empty(max(plan.workspace(), 16), dtype=torch.uint8, device=DEV))
        return y
    check(call, act, float("nan"))
