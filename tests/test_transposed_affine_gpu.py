"""Binary-weight affine layers and input gradients whose product runs with the weights on the MMA rows: shapes at the
edges of its 128 x 64 tiles, with rows that 128-bit accesses do not fit, alpha made from partial sums, accumulation."""
import pytest
import torch

from launches import kernels

pytestmark = pytest.mark.gpu

# (rows, inmaps, outmaps): past the sizes of the one-launch products
SHAPES = [(256, 1024, 4096), (63, 4100, 129), (65, 2048, 700), (129, 3000, 1027), (1, 8192, 513), (300, 1111, 2050)]


@pytest.mark.parametrize("M,K,N", SHAPES)
def test_forward_and_input_gradient(M, K, N):
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, b, dy = r(M, K), r(K, N), r(N), r(M, N)
    wb, alpha = torch.zeros_like(w), torch.zeros(N, device="cuda")
    y = F.binary_weight_affine(x, w, wb, alpha, b)
    sign = torch.where(w > 0, 1.0, torch.where(w < 0, -1.0, 1.0))
    a = w.double().abs().mean(0)
    assert torch.equal(wb, sign)
    # sums of K positive values, fp32
    assert ((alpha.double() - a).abs() <= 4 * 2.0 ** -24 * K ** 0.5 * a).all()
    # the tensor core's sums: 1.4e-6 of the result's root mean square however long they are, three times that
    rms = lambda t: t.square().mean().sqrt()
    want = (x.double() @ sign.double()) * a + b.double()
    assert rms(y.double() - want) <= 4.2e-6 * rms(want)
    connect = F.binary_connect_affine(x, w, torch.zeros_like(w), b)
    want = x.double() @ sign.double() + b.double()
    assert rms(connect.double() - want) <= 4.2e-6 * rms(want)
    old = torch.ones_like(x)
    dx = F.binary_weight_affine_backward(x, wb, alpha, dy, propagate_down=(True, False, False))[0]
    want = (dy.double() * alpha.double()) @ sign.double().t()
    assert rms(dx.double() - want) <= 4.2e-6 * rms(want)
    acc = F.binary_weight_affine_backward(x, wb, alpha, dy, propagate_down=(True, False, False),
                                          accum=(True, False, False), grads=(old, None, None))[0]
    assert torch.equal(acc, dx + 1.0)


# Around the line to the two-SM kernel, which makes no alpha: 148 SMs take 74 of its 256 x 256 tiles, while 147 of 128 x 128
# leave one of them idle. On either side of it in outputs, in rows and in the length of K; bias and no bias.
@pytest.mark.parametrize("M,K,N,last", [
    (64, 1024, 18704, "gemm_pair_tcgen05"), (128, 512, 18816, "gemm_pair_tcgen05"), (128, 512, 18820, "gemm_pair_tcgen05"),
    (64, 2048, 18692, "gemm_pair_tcgen05"), (64, 1022, 18704, "gemm_pair_tcgen05"), (18816, 256, 100, "gemm_pair_tcgen05"),
    (18689, 512, 128, "gemm_pair_tcgen05"), (64, 2052, 18692, "gemm_tcgen05_transposed"),
    (128, 512, 18688, "gemm_tcgen05_transposed"), (64, 1024, 18702, "gemm_tcgen05_transposed"),
    (18688, 256, 100, "gemm_tcgen05_transposed")])
@pytest.mark.parametrize("bias", [True, False])
def test_alpha_at_the_line_to_the_two_sm_kernel(M, K, N, last, bias):
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w, b = r(M, K), r(K, N), r(N) if bias else None
    wb, alpha = torch.zeros_like(w), torch.full((N,), -1.0, device="cuda")
    y = F.binary_weight_affine(x, w, wb, alpha, b)
    a = w.double().abs().mean(0)
    assert ((alpha.double() - a).abs() <= 4 * 2.0 ** -24 * K ** 0.5 * a).all()
    sign = torch.where(w < 0, -1.0, 1.0)  # (a few of the many normal values are zero)
    want = (x.double() @ sign.double()) * a + (b.double() if bias else 0.0)
    # a whole tile's sums in tensor memory: 2.6e-6 of the root mean square at K = 1024, growing with K up to 2048
    rms = lambda t: t.square().mean().sqrt()
    assert rms(y.double() - want) <= 1e-5 * rms(want)
    taken = kernels(lambda: F.binary_weight_affine(x, w, wb, alpha, b))
    print(*taken)
    assert taken[-1] == last
