"""Inference batch normalisation and the activation operator by four elements at a time: planes that are and are not multiples of
four, counts with a remainder, unaligned tensors, in place -- against the formula in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from gpu_util import DEV


@pytest.mark.parametrize("batch,features,plane", [(1, 1, 1), (2, 3, 49), (3, 5, 4), (1, 7, 3), (2, 64, 196), (5, 33, 13 * 13), (16, 256, 56 * 56)])
@pytest.mark.parametrize("offset,affine,in_place", [(0, True, False), (1, True, True), (0, False, True)])
def test_batchnorm(batch, features, plane, offset, affine, in_place):
    from dlprimitives_b200 import capi
    g = torch.Generator(device=DEV).manual_seed(plane)
    count = batch * features * plane
    x = torch.randn(count + offset, device=DEV, generator=g)[offset:].view(batch, features, plane, 1)
    y = x if in_place else torch.full((count + offset,), float("nan"), device=DEV)[offset:].view(batch, features, plane, 1)
    mean, gamma, beta = (torch.randn(features, device=DEV, generator=g) for _ in range(3))
    var = torch.rand(features, device=DEV, generator=g) + 0.1
    # in 64 bits: a and b are each within 3 roundings of theirs, the product and the sum add two more
    a = 1.0 / (var.double() + 1e-5).sqrt() * (gamma.double() if affine else 1.0)
    want = x.double() * a[None, :, None, None] + (-mean.double() * a + (beta.double() if affine else 0.0))[None, :, None, None]
    bound = 6 * 2.0 ** -24 * (x.double().abs() * a.abs()[None, :, None, None] + (mean.double() * a).abs()[None, :, None, None] + beta.double().abs()[None, :, None, None])
    capi.batchnorm_inference(x, y, mean, var, gamma if affine else None, beta if affine else None, eps=1e-5)
    assert bool(((y.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("count", [1, 3, 4, 1023, 100000])
@pytest.mark.parametrize("offset", [0, 1])
def test_activation(count, offset):
    from dlprimitives_b200 import capi
    x = torch.randn(count + offset, device=DEV, generator=torch.Generator(device=DEV).manual_seed(count))[offset:]
    y = torch.full((count + offset,), float("nan"), device=DEV)[offset:]
    capi.activation(x, y, "relu6")
    assert torch.equal(y, x.clamp(0.0, 6.0))
    want = torch.relu(x)
    capi.activation(x, x, "relu")
    assert torch.equal(x, want)
