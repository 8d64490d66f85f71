"""Batch normalization's sums over a channel where a channel has several blocks, with one and several sets of loads per
thread, aligned and not, and more channels than a round of blocks: against 64-bit sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 16, 56, 56), (64, 37, 29, 31), (2, 1300, 4, 4), (40, 600, 7, 7), (9, 1, 64, 64)])
def test_statistics_and_parameter_gradients(shape):
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    C, count = shape[1], shape[0] * shape[2] * shape[3]
    x = torch.randn(*shape, device="cuda", generator=g).mul_(2.0).add_(0.7)
    dy = torch.randn(*shape, device="cuda", generator=g).add_(0.05)
    full = lambda v: torch.full((1, C, 1, 1), v, device="cuda")
    _, mean, var = F.batch_normalization(x, full(0.1), full(1.1), full(0.0), full(1.0), [1], 0.9, 1e-5, True,
                                         output_stat=True)
    _, dbeta, dgamma = F.batch_normalization_backward(x, dy, full(1.1), mean, var)
    rows = lambda t: t.double().transpose(0, 1).reshape(C, -1)
    xd, gd = rows(x), rows(dy)
    md, vd = xd.mean(1), xd.var(1, unbiased=False)
    xh = (xd - md[:, None]) / (vd[:, None] + 1e-5).sqrt()
    # a sum is off by at most a few roundings of the size of its terms' root sum of squares; x^2 - mean^2 cancels a little
    # (var is 4, the terms 4.5), and the gradients use the rounded mean and variance
    for got, want, terms in ((mean, md, xd / count), (var, vd, xd * xd / count), (dbeta, gd.sum(1), gd),
                             (dgamma, (gd * xh).sum(1), gd * xh)):
        size = terms.square().sum(1).sqrt() + want.abs()
        assert ((got.double().reshape(-1) - want).abs() <= 16 * 2.0 ** -24 * size * max(1.0, (count / 4096) ** 0.5)).all()
