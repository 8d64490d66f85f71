"""GPU parity of the quantizers' backward passes, through the C ABI: input
gradients bit-exact against the golden vectors made by the reference's own
Function::backward and against the oracle on sizes that exercise the
vector body, tails and misaligned buffers; the two range gradients of
MinMaxQuantize (fp32 sums) to rounding."""
import numpy as np
import pytest
import torch

import backward_cases
import cases
from golden_util import bits
from oracle import oracle

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def host(t):
    return t.cpu().numpy()


@pytest.fixture(scope="module")
def F():
    from nnabla_b200 import _capi, functions
    _capi.call("nb200_check_device")
    return functions


class Device:
    """The CUDA path behind the oracle's numpy signatures."""

    def __init__(self, F):
        self.F = F

    def fixed_point_quantize_backward(self, x, dy, sign, n, delta, fine, accum, dx0):
        return host(self.F.fixed_point_quantize_backward(dev(x), dev(dy), sign, n, delta, fine, accum, dev(dx0)))

    def pow2_quantize_backward(self, x, dy, sign, wz, n, m, fine, accum, dx0):
        return host(self.F.pow2_quantize_backward(dev(x), dev(dy), sign, wz, n, m, fine, accum, dev(dx0)))

    def min_max_quantize(self, x, qmin, qmax, lmin, lmax, decay, xmm, ema, eps):
        a, b = dev(qmin), dev(qmax)
        y = self.F.min_max_quantize(dev(x), a, b, dev(lmin), dev(lmax), decay, xmm, ema, True, eps)
        return host(y), host(a), host(b)

    def min_max_quantize_backward(self, x, qmin, qmax, lmin, lmax, dy, xmm, ema, fine, pd, ac, g0):
        r = self.F.min_max_quantize_backward(dev(x), dev(qmin), dev(qmax), dev(lmin), dev(lmax), dev(dy), xmm, ema,
                                             fine, pd, ac, [dev(g) for g in g0])
        return tuple(host(t) for t in r)


@pytest.mark.parametrize("i", range(len(cases.FXP_GRID)))
@pytest.mark.parametrize("fine,accum", backward_cases.FLAGS)
def test_fxp_backward_golden(F, i, fine, accum):
    backward_cases.check_fxp(Device(F), i, fine, accum)


@pytest.mark.parametrize("i", range(len(backward_cases.POW2_CASES)))
@pytest.mark.parametrize("fine,accum", backward_cases.FLAGS)
def test_pow2_backward_golden(F, i, fine, accum):
    backward_cases.check_pow2(Device(F), i, fine, accum)


@pytest.mark.parametrize("i", range(len(cases.MINMAX_GRID)))
@pytest.mark.parametrize("fine,accum", backward_cases.FLAGS)
def test_minmax_backward_golden(F, i, fine, accum):
    backward_cases.check_minmax(Device(F), i, fine, accum)


@pytest.mark.parametrize("size", cases.VEC_TAIL_SIZES + [1 << 20])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("accum", [False, True])
def test_backward_tails_and_misalignment(F, size, offset, accum):
    rng = np.random.RandomState(size + offset)
    x = (rng.randn(size + offset) * 6).astype(np.float32)
    dy = rng.randn(size + offset).astype(np.float32)
    dx0 = rng.randn(size + offset).astype(np.float32)
    xd, dyd = dev(x)[offset:], dev(dy)[offset:]
    sl = slice(offset, None)
    got = F.fixed_point_quantize_backward(xd, dyd, True, 8, 2.0 ** -4, True, accum, dev(dx0)[offset:].contiguous())
    want = oracle.fixed_point_quantize_backward(x[sl], dy[sl], True, 8, 2.0 ** -4, True, accum, dx0[sl])
    assert np.array_equal(bits(host(got)), bits(want))
    got = F.pow2_quantize_backward(xd, dyd, True, True, 8, 1, True, accum, dev(dx0)[offset:].contiguous())
    want = oracle.pow2_quantize_backward(x[sl], dy[sl], True, True, 8, 1, True, accum, dx0[sl])
    assert np.array_equal(bits(host(got)), bits(want))
    got = F.pow2_quantize_backward(xd, dyd, False, False, 4, 0, False, accum, dev(dx0)[offset:].contiguous())
    want = oracle.pow2_quantize_backward(x[sl], dy[sl], False, False, 4, 0, False, accum, dx0[sl])
    assert np.array_equal(bits(host(got)), bits(want))


def test_pow2_backward_extreme_ranges(F):
    """p_max beyond every float (no gradient is blocked) and below every float
    (every non-zero input is blocked)."""
    x = np.concatenate([cases.edge_values_pow2(), np.array([np.nan, 0.0, -0.0], np.float32)])
    dy, dx0 = cases.grad_inputs(x)
    for m in (200, 128, 127, -140, -149, -150, -300):
        want = oracle.pow2_quantize_backward(x, dy, True, True, 4, m, True, False, dx0)
        got = F.pow2_quantize_backward(dev(x), dev(dy), True, True, 4, m, True, False)
        assert np.array_equal(bits(host(got)), bits(want)), m


def test_minmax_backward_large_per_tensor(F):
    """BASELINE configs[1] ranges on 2^22 elements: dx bit-exact, range gradients against a float64 sum."""
    rng = np.random.RandomState(0)
    n = 1 << 22
    x = rng.uniform(-4.5, 4.5, n).astype(np.float32)
    dy = rng.randn(n).astype(np.float32)
    one = lambda v: np.array([v], np.float32)
    qmin, qmax, lmin, lmax = one(-4), one(4), one(0), one(255)
    _, fmin, fmax, _ = oracle.min_max_quantize(x, qmin, qmax, lmin, lmax)
    want_dx, _, _ = oracle.min_max_quantize_backward(x, fmin, fmax, lmin, lmax, dy)
    dx, gmin, gmax = F.min_max_quantize_backward(dev(x), dev(fmin), dev(fmax), dev(lmin), dev(lmax), dev(dy))
    assert np.array_equal(bits(host(dx)), bits(want_dx))
    # nudged range (min_max_quantize.cpp:362-390) in fp32: scale 8/255, zero point round(0 - (-4 / scale)) = 127
    scale = np.float32(8) / np.float32(255)
    zp = np.round(np.float32(0) - np.float32(-4) / scale)
    m, M = (np.float32(0) - zp) * scale, (np.float32(255) - zp) * scale
    lo64 = dy[x < m].astype(np.float64).sum()
    hi64 = dy[x > M].astype(np.float64).sum()
    assert abs(float(host(gmin)[0]) - lo64) < 1e-3 and abs(float(host(gmax)[0]) - hi64) < 1e-3


def test_backward_argument_errors(F):
    x = torch.zeros(8, device="cuda")
    with pytest.raises(RuntimeError):
        F.fixed_point_quantize_backward(x, torch.zeros(9, device="cuda"))
    with pytest.raises(RuntimeError):
        F.fixed_point_quantize_backward(x, x, accum=True)
    with pytest.raises(RuntimeError):
        F.fixed_point_quantize_backward(x, x, n=0)
    with pytest.raises(RuntimeError):
        F.pow2_quantize_backward(x, x, n=1)


# one block per range up to 8192 elements, the launches of separate steps above
@pytest.mark.parametrize("shape,axis", [((1, 1, 1), None), ((3, 5, 7), 1), ((2, 3, 4097), 1), ((8, 24, 1024), 1),
                                        ((8, 24, 1025), 1), ((8192,), None), ((8193,), None), ((700, 2), 0)])
@pytest.mark.parametrize("observe", [True, False])
@pytest.mark.parametrize("fine", [True, False])
def test_min_max_quantize_range_lengths(shape, axis, observe, fine):
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(len(shape))
    x, dy = (torch.randn(*shape, device="cuda", generator=g) * 3 for _ in range(2))
    qshape = [n if i == axis else 1 for i, n in enumerate(shape)]
    dims = [i for i in range(len(shape)) if i != axis]
    qmin, qmax = torch.full(qshape, -1.5, device="cuda"), torch.full(qshape, 2.0, device="cuda")
    lmin, lmax = torch.zeros(qshape, device="cuda"), torch.full(qshape, 255.0, device="cuda")
    y = F.min_max_quantize(x, qmin, qmax, lmin, lmax, x_min_max=observe)
    lo, hi = (x.amin(dims, keepdim=True), x.amax(dims, keepdim=True)) if observe else (qmin, qmax)
    hi = torch.where(hi - lo < 0.01, lo + 0.01, hi)
    assert torch.equal(qmin, lo) and torch.equal(qmax, hi)
    s = (hi - lo) / 255
    zp = torch.clamp(torch.round(-lo / s), 0, 255)
    m, M = -zp * s, (255 - zp) * s
    assert ((y - (torch.round((torch.minimum(torch.maximum(x, m), M) - m) / s) * s + m)).abs() <= 1.01 * s).all()
    old = torch.ones_like(x)
    for accum, buffer in ((False, None), (True, old)):
        dx, g_lo, g_hi = F.min_max_quantize_backward(x, qmin, qmax, lmin, lmax, dy, x_min_max=observe, ste_fine_grained=fine,
                                                     accum=(accum, False, False), grads=(buffer, None, None))
        inside = (x >= m) & (x <= M) if fine else torch.ones_like(x, dtype=torch.bool)
        off = dx - float(accum) - dy * inside
        assert (off.abs() <= 1e-6 * (1 + dy.abs())).float().mean() >= 1 - 3 / x.numel()  # a bound itself may round
        for got, side in ((g_lo, x < m), (g_hi, x > M)):
            want = torch.zeros_like(got) if observe else (dy.double() * side).sum(dims, keepdim=True)
            assert got.shape == torch.Size(qshape) and ((got - want).abs() <= 1e-4 * dy.abs().sum() ** 0.5 + 1e-5).all()


def _kernels(fn):
    """Kernel launches of fn, from its CUDA graph."""
    from cuda.bindings import runtime
    fn()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        fn()
    graph = runtime.cudaGraph_t(g.raw_cuda_graph())
    _, _, count = runtime.cudaGraphGetNodes(graph)
    err, nodes, _ = runtime.cudaGraphGetNodes(graph, count)
    assert err == runtime.cudaError_t.cudaSuccess
    return sum(runtime.cudaGraphNodeGetType(n)[1] == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel
               for n in nodes[:count])


# the lines of minmax_one_block: (forward, observed, gradient) in one launch
@pytest.mark.parametrize("shape,one", [
    ((16, 24, 49), (True, True, True)),          # an activation, a range per channel
    ((1, 1, 4096), (True, True, True)),
    ((1, 1, 8192), (False, True, True)),         # a single long range
    ((1, 1, 8193), (False, False, False)),
    ((1024, 256, 1), (True, True, True)),        # weights with a range per output column: a small matrix
    ((1024, 257, 1), (False, False, False)),
    ((2049, 16, 1), (False, False, False)),
    ((1024, 512, 2), (True, True, True)),
    ((1024, 513, 2), (False, False, False)),
    ((4096, 4096, 1), (False, False, False)),
    ((1024, 256, 4), (True, True, True)),        # runs of 16 bytes
    ((2, 1024, 3), (True, True, True)),          # many ranges
    ((2, 1025, 3), (False, False, False)),
    ((4, 4096, 256), (True, True, True)),
    ((5, 4096, 256), (True, True, False)),
    ((4, 4097, 256), (False, False, False)),
    ((1, 65536, 4), (False, True, None)),        # more ranges than the reduction over the whole tensor takes
])
def test_min_max_quantize_route(F, shape, one):
    """Each call takes the form that was measured to be the faster one, and both give the oracle's bits."""
    rng = np.random.RandomState(shape[1])
    x = rng.uniform(-4.5, 4.5, shape).astype(np.float32)
    dy = rng.randn(*shape).astype(np.float32)
    q = [np.full((1, shape[1], 1), v, np.float32) for v in (-4.0, 4.0, 0.0, 255.0)]
    gx, gdy, r = dev(x), dev(dy), [dev(v) for v in q]
    for observe in (False, True):
        want, lo, hi, _ = oracle.min_max_quantize(x, *q, 0.9, observe, observe)
        mine = [t.clone() for t in r]
        got = F.min_max_quantize(gx, *mine, 0.9, observe, observe)
        for a, b in ((got, want), (mine[0], lo), (mine[1], hi)):
            assert np.array_equal(bits(host(a)), bits(b))
        assert (_kernels(lambda: F.min_max_quantize(gx, *mine, 0.9, observe, observe)) == 1) == one[int(observe)]
    if one[2] is None:
        with pytest.raises(RuntimeError, match="65535"):
            F.min_max_quantize_backward(gx, *r, gdy, x_min_max=True)
        return
    want, _, _ = oracle.min_max_quantize_backward(x, *q, dy, True, True)
    got, glo, ghi = F.min_max_quantize_backward(gx, *r, gdy, x_min_max=True, ema=True)
    assert np.array_equal(bits(host(got)), bits(want)) and not glo.any() and not ghi.any()
    assert (_kernels(lambda: F.min_max_quantize_backward(gx, *r, gdy, x_min_max=True, ema=True)) == 1) == one[2]
