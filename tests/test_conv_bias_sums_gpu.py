"""Bias gradients of convolutions: sums taken by the pass that converts dy (up to 1024 tiles of 64 pixels) and by a pass of
their own, images of whole and ragged tiles, groups, fewer and more maps than a tile, accumulation: against 64-bit sums.
Channels that are no multiple of the weights' slots, whose other slots are zero."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,cin,maps,height,width,group", [(3, 16, 24, 8, 8, 1), (2, 20, 70, 13, 7, 1), (24, 8, 160, 35, 29, 1),
                                                               (22, 16, 16, 56, 56, 1), (5, 24, 36, 9, 11, 2), (1, 16, 9, 3, 5, 1)])
@pytest.mark.parametrize("accum", [False, True])
def test_bias_gradient(batch, cin, maps, height, width, group, accum):
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(maps)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, dy = r(batch, cin, height, width), r(maps, cin // group, 3, 3), r(batch, maps, height, width).add_(0.1)
    wb = torch.zeros_like(w)
    y = F.binary_connect_convolution(x, w, wb, None, 1, (1, 1), (1, 1), group=group)
    want = torch.nn.functional.conv2d(x.double(), wb.double(), None, 1, 1, 1, group)
    assert (y.double() - want).square().mean().sqrt() <= 4e-6 * want.square().mean().sqrt()
    old = torch.ones(maps, device="cuda")
    grads = F.binary_connect_convolution_backward(x, wb, dy, 1, (1, 1), (1, 1), group=group, accum=(False, False, accum),
                                                  grads=(None, None, old.clone() if accum else None))
    want = dy.double().sum((0, 2, 3)) + (1.0 if accum else 0.0)
    size = dy.double().square().sum((0, 2, 3)).sqrt() + want.abs()
    # a few roundings of partial sums no larger than a few times the root sum of squares
    assert ((grads[2].double() - want).abs() <= 16 * 2.0 ** -24 * size).all()
