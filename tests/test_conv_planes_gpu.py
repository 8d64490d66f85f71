"""Convolution gradients at the edges of the pixel-major kernels (boxes, tap groups, classes of a stride, channel and
map blocks) against float64 convolutions: dx and dW within 1e-5 of their RMS."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# batch, channels, height, width, maps, kernel, pad, stride, dilation, group
CASES = [
    (1, 64, 64, 64, 64, 3, 1, 1, 1, 1),     # the widest rows of a box
    (2, 130, 13, 61, 70, 3, 1, 1, 1, 1),    # several channel and map blocks, ragged rows
    (3, 48, 11, 9, 40, 5, 2, 1, 1, 1),      # 25 taps: seven tap groups
    (5, 16, 29, 31, 200, 3, 1, 2, 1, 1),    # four classes of a stride, two column tiles
    (2, 20, 23, 17, 33, 3, 2, 3, 2, 1),     # classes without taps
    (4, 96, 10, 10, 64, 1, 0, 2, 1, 1),     # one tap, three empty classes
    (2, 72, 14, 15, 136, 3, 0, 1, 1, 2),    # groups whose slots are padded
    (300, 8, 3, 3, 8, 3, 1, 1, 1, 1),       # many tiny images
    (80, 128, 27, 27, 256, 1, 0, 2, 1, 1),  # a tile with more boxes than the ring, several tiles per block
    (1, 24, 7, 120, 16, 3, 1, 1, 1, 1),     # rows near the width limit
]


@pytest.mark.parametrize("n,c,h,w,o,k,pad,stride,dil,group", CASES)
@pytest.mark.parametrize("delta", [None, 2.0 ** -4])
def test_gradients(n, c, h, w, o, k, pad, stride, dil, group, delta):
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(n + c)
    x = torch.randn(n, c, h, w, device="cuda", generator=g)
    if delta:
        x = (x / delta).round().clamp(-127, 127) * delta
    wb = torch.randn(o, c // group, k, k, device="cuda", generator=g).sign()
    alpha = torch.rand(o, device="cuda", generator=g) + 0.5
    geometry = dict(pad=(pad, pad), stride=(stride, stride), dilation=(dil, dil), group=group)
    xd, wd = x.double().requires_grad_(), (wb.double() * alpha.double().view(-1, 1, 1, 1)).requires_grad_()
    y = torch.nn.functional.conv2d(xd, wd, None, stride, pad, dil, group)
    dy = torch.randn(*y.shape, device="cuda", generator=g)
    y.backward(dy.double())
    dx, dw, db = F.binary_weight_convolution_backward(x, wb, alpha, dy, fixed_point_delta=delta, **geometry)
    dx0, dw0 = torch.ones_like(x), torch.ones_like(wb)
    F.binary_weight_convolution_backward(x, wb, alpha, dy, propagate_down=(True, True, False), accum=(True, True, False),
                                         grads=(dx0, dw0, None), fixed_point_delta=delta, **geometry)
    F.check_device_status()
    for got, want in ((dx, xd.grad), (dw, wd.grad), (dx0 - 1, xd.grad), (dw0 - 1, wd.grad), (db, dy.double().sum((0, 2, 3)))):
        assert (got.double() - want).norm() <= 1e-5 * want.norm() + 1e-6 * want.numel() ** 0.5


@pytest.mark.parametrize("n,c,h,w,o,k,pad,stride,dil,group", CASES)
def test_forward(n, c, h, w, o, k, pad, stride, dil, group):
    """Images of very different magnitudes: each has a scale of its own."""
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(n + c)
    x = torch.randn(n, c, h, w, device="cuda", generator=g)
    x *= torch.exp2(torch.randint(-30, 30, (n, 1, 1, 1), device="cuda", generator=g).float())
    wt = torch.randn(o, c // group, k, k, device="cuda", generator=g)
    wb, alpha = torch.empty_like(wt), torch.empty(o, device="cuda")
    y = F.binary_weight_convolution(x, wt, wb, alpha, None, 1, (pad, pad), (stride, stride), (dil, dil), group)
    F.check_device_status()
    want = torch.nn.functional.conv2d(x.double(), wb.double() * alpha.double().view(-1, 1, 1, 1), None, stride, pad, dil, group)
    error = (y.double() - want).flatten(1).norm(dim=1) / want.flatten(1).norm(dim=1)
    assert error.max() <= 2e-6


# batch, channels, height, width, maps, kernel, pad, stride, group; blocks of the forward and of the input gradient: a
# tile each, up to one per SM
SMALL = [
    (64, 96, 7, 7, 512, 3, 1, 1, 1, 128, 64),       # two images a tile, a box per filter row; one round as it is
    (75, 512, 8, 8, 200, 3, 1, 1, 1, 76, 148),      # a box per tap; one image in the last tile
    (400, 130, 5, 5, 64, 3, 1, 1, 1, 134, 148),     # three images a tile; 64 columns
    (100, 256, 7, 7, 130, 1, 0, 1, 1, 100, 100),    # no halo
    (100, 64, 13, 15, 130, 3, 1, 2, 1, 100, 148),   # a stride: classes of taps, and of pixels
    (90, 128, 6, 6, 256, 3, 1, 1, 2, 90, 90),       # groups
    (700, 512, 2, 2, 128, 3, 1, 1, 1, 44, 88),      # many images a tile
    (30, 300, 9, 8, 300, 5, 2, 2, 1, 90, 96),       # classes of 5 x 4 pixels and fewer
    (50, 260, 9, 9, 200, 1, 0, 2, 1, 100, 120),     # three classes that no tap reaches
]


def _blocks(fn):
    """Blocks of the pixel-major kernel (the one with 352 threads) in fn, from its CUDA graph."""
    from cuda.bindings import driver
    fn()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    graph = driver.CUgraph(g.raw_cuda_graph())
    _, _, count = driver.cuGraphGetNodes(graph)
    _, nodes, _ = driver.cuGraphGetNodes(graph, count)
    kernel = driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL
    params = [driver.cuGraphKernelNodeGetParams(n)[1] for n in nodes[:count] if driver.cuGraphNodeGetType(n)[1] == kernel]
    return [p.gridDimX for p in params if p.blockDimX == 352]


@pytest.mark.parametrize("n,c,h,w,o,k,pad,stride,group,blocks,blocks_dx", SMALL)
def test_small_images_share_tiles(n, c, h, w, o, k, pad, stride, group, blocks, blocks_dx):
    """Images of at most 64 pixels, of very different magnitudes: several in a tile where that takes fewer rounds."""
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(n + c)
    x = torch.randn(n, c, h, w, device="cuda", generator=g)
    x *= torch.exp2(torch.randint(-30, 30, (n, 1, 1, 1), device="cuda", generator=g).float())
    wt = torch.randn(o, c // group, k, k, device="cuda", generator=g)
    wb, alpha = torch.empty_like(wt), torch.empty(o, device="cuda")
    b = torch.randn(o, device="cuda", generator=g)
    geometry = dict(pad=(pad, pad), stride=(stride, stride), group=group)
    forward = lambda bias: F.binary_weight_convolution(x, wt, wb, alpha, bias, **geometry)
    y, yb = forward(None), forward(b)
    assert torch.equal(yb, y + b.view(1, -1, 1, 1))
    xd, wd = x.double().requires_grad_(), wb.double() * alpha.double().view(-1, 1, 1, 1)
    want = torch.nn.functional.conv2d(xd, wd, None, stride, pad, 1, group)
    per_image = lambda got, ref: (got.double() - ref).flatten(1).norm(dim=1) / ref.flatten(1).norm(dim=1)
    assert per_image(y, want.detach()).max() <= 2e-6
    dy = torch.randn(*y.shape, device="cuda", generator=g)
    dy *= torch.exp2(torch.randint(-30, 30, (n, 1, 1, 1), device="cuda", generator=g).float())
    want.backward(dy.double())
    gradient = lambda **kw: F.binary_weight_convolution_backward(x, wb, alpha, dy, propagate_down=(True, False, False),
                                                                 **geometry, **kw)[0]
    dx = gradient()
    assert per_image(dx, xd.grad).max() <= 2e-6
    old = torch.randn(*x.shape, device="cuda", generator=g)
    assert torch.equal(gradient(accum=(True, False, False), grads=(old.clone(), None, None)), old + dx)
    F.check_device_status()
    assert _blocks(lambda: forward(b)) == [blocks] and _blocks(gradient) == [blocks_dx]


@pytest.mark.parametrize("n,c,h,w,o,k,pad,stride,dil,group", CASES[:6] + CASES[7:8])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_weight_gradient_of_values_that_are_not_finite(n, c, h, w, o, k, pad, stride, dil, group, bad):
    """A value of x that is not finite reaches the taps that pair it with an output pixel, and no others."""
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(n + c)
    x = torch.randn(n, c, h, w, device="cuda", generator=g)
    x[0, 0, 0, 0] = x[-1, c - 1, h - 1, w - 1] = x[0, c // 2, h // 2, w - 1] = bad
    wb = torch.randn(o, c // group, k, k, device="cuda", generator=g).sign()
    geometry = dict(pad=(pad, pad), stride=(stride, stride), dilation=(dil, dil), group=group)
    dy = torch.randn_like(F.binary_connect_convolution(x, wb, torch.empty_like(wb), **geometry))
    gradient = lambda **kw: F.binary_connect_convolution_backward(x, wb, dy, propagate_down=(False, True, False),
                                                                  **geometry, **kw)[1]
    # the taps one by one: the pixels of x that each pairs with dy, zeros outside the image
    xp = torch.nn.functional.pad(x.double(), (pad,) * 4)
    want = torch.empty(o, c // group, k, k, dtype=torch.float64, device="cuda")
    for ky in range(k):
        for kx in range(k):
            part = xp[:, :, ky * dil:ky * dil + (dy.shape[2] - 1) * stride + 1:stride,
                      kx * dil:kx * dil + (dy.shape[3] - 1) * stride + 1:stride]
            for i in range(group):
                a = dy.double().chunk(group, 1)[i].transpose(0, 1).flatten(1)
                b = part.chunk(group, 1)[i].transpose(0, 1).flatten(1)
                want.chunk(group, 0)[i][:, :, ky, kx] = a @ b.t()
    got = gradient()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isposinf(), want.isposinf())
    finite = want.isfinite()
    assert (got.double() - want)[finite].norm() <= 1e-5 * want[finite].norm() and not finite.all() and finite.any()
    assert torch.equal(gradient(accum=(False, True, False), grads=(None, torch.ones_like(wb), None)).isnan(), want.isnan())
    F.check_device_status()
