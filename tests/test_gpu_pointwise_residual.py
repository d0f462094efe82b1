"""The 1x1 kernel with a fused residual at the channel counts where its shared memory is shared out differently: every number of
k-blocks over 64-channel tiles, and the other tiles at their ends -- against the same layer in 64 bits, several passes each."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_util import DEV

# as in test_gpu_stream.py: 3xTF32 terms within 2^-21, sums of eight k-blocks truncated at 2^-23 a step
TOL = 5e-6


@pytest.mark.parametrize("cin,cout", [(32 * k, 64) for k in range(1, 9)] + [(224, 40), (200, 33), (224, 128), (32, 32), (256, 32), (64, 256)])
def test_residual(cin, cout):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(cin + cout)
    batch, hw = 20, 56
    x = torch.randn(batch, cin, hw, hw, device=DEV, generator=g)
    w = torch.randn(cout, cin, 1, 1, device=DEV, generator=g) * (2.0 / cin) ** 0.5
    bias = torch.randn(cout, device=DEV, generator=g)
    res = torch.randn(batch, cout, hw, hw, device=DEV, generator=g)
    plan = capi.Conv2DForward(channels_in=cin, channels_out=cout, kernel=1, batch=batch, height=hw, width=hw, bias=True)
    packed = plan.prepack(w)
    ws = torch.empty(max(plan.workspace(), 16), dtype=torch.uint8, device=DEV)
    y = torch.full_like(res, float("nan"))
    want = torch.matmul(w.double().reshape(cout, cin), x.double().reshape(batch, cin, -1)).reshape(res.shape)
    want = torch.relu(want + bias.double()[None, :, None, None] + res.double())
    for _ in range(4):
        plan.enqueue_packed(x, packed, bias, y, residual=res, post_activation="relu", ws=ws)
        assert capi.device_status() == 0
        assert float((y.double() - want).norm() / want.norm()) < TOL
