"""Small affine products on the FMA pipes: both gradients in one launch against each in its own (the same tiles, so the
same bits) and against 64-bit sums; binarized weights written by all blocks of a column. Sizes at the edges of the 16 and
32 row tiles, of the 128-value chunks and of their 16-value shares, with rows that are not 16-byte aligned."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (1, 130, 33), (16, 32, 128), (17, 129, 31), (100, 784, 500), (33, 1025, 70), (130, 500, 96),
          (65, 300, 1000), (300, 1000, 200)]


def data(M, K, N):
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    return r(M, K), r(K, N), r(N), r(M, N)


@pytest.mark.parametrize("M,K,N", SHAPES)
@pytest.mark.parametrize("accum", [False, True])
def test_gradients_in_one_launch(M, K, N, accum):
    from nnabla_b200 import functions as F
    x, w, b, dy = data(M, K, N)
    wb, alpha = torch.zeros_like(w), torch.zeros(N, device="cuda")
    F.binary_weight_affine(x, w, wb, alpha, b)
    old = [torch.ones_like(x), torch.ones_like(w), torch.ones_like(b)]

    def grads(*down):
        into = [t.clone() if accum and d else None for t, d in zip(old, down)]
        return F.binary_weight_affine_backward(x, wb, alpha, dy, propagate_down=down,
                                               accum=tuple(accum and d for d in down), grads=tuple(into))
    dx, dw, db = grads(True, True, True)
    assert torch.equal(dx, grads(True, False, False)[0])
    dw1, db1 = grads(False, True, True)[1:]
    assert torch.equal(dw, dw1) and torch.equal(db, db1)
    add = 1.0 if accum else 0.0
    wants = [(dy.double() * alpha.double()) @ wb.double().t() + add, x.double().t() @ dy.double() + add,
             dy.double().sum(0) + add]
    for got, want in zip((dx, dw, db), wants):
        # fp32 sums of up to K values in at most 2^-24 * sqrt(K) relative to their root mean square, times four
        bound = 4 * 2.0 ** -24 * max(M, N, 16) ** 0.5
        scale = want.square().mean().sqrt()
        assert (got.double() - want).square().mean().sqrt() <= bound * scale


@pytest.mark.parametrize("M,K,N", SHAPES)
def test_binarized_weights_come_from_every_block(M, K, N):
    from nnabla_b200 import functions as F
    x, w, b, _ = data(M, K, N)
    w[0, 0] = 0.0
    wb, alpha = torch.full_like(w, 7.0), torch.zeros(N, device="cuda")
    y = F.binary_weight_affine(x, w, wb, alpha, b)
    sign = torch.where(w > 0, 1.0, torch.where(w < 0, -1.0, 1.0))
    assert torch.equal(wb, sign)
    a = w.double().abs().mean(0)
    assert ((alpha.double() - a).abs() <= 4 * 2.0 ** -24 * K ** 0.5 * a).all()
    want = (x.double() @ sign.double()) * alpha.double() + b.double()
    assert (y.double() - want).square().mean().sqrt() <= 4 * 2.0 ** -24 * K ** 0.5 * want.square().mean().sqrt()
