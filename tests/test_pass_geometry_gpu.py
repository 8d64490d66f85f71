"""Elementwise passes at the edges of their launches: one vector a thread below 148 * 4 * 256 of them, four above, whole
and ragged last blocks, remainders of a vector, tensors off the 16-byte grid, results that are stored streaming. Each
value is compared bit for bit with the oracle, so a run that is missed, doubled or moved shows."""
import numpy as np
import pytest
import torch

from golden_util import bits
from oracle import oracle

pytestmark = pytest.mark.gpu

FEW = 148 * 4 * 256 * 4  # values up to which a thread takes one vector
SIZES = [1, 3, 1023, 1025, 4096, FEW, FEW + 1, FEW + 5, FEW + 4096 + 7]


@pytest.fixture(scope="module")
def F():
    from nnabla_b200 import _capi, functions
    _capi.call("nb200_check_device")
    return functions


def same(t, a):
    return np.array_equal(bits(t.cpu().numpy().reshape(-1)), bits(np.asarray(a, np.float32).reshape(-1)))


def tensor(a, offset=0):
    t = torch.empty(a.size + offset, device="cuda")[offset:]
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("size", SIZES)
def test_elementwise(F, size, offset):
    rng = np.random.RandomState(size % 1000)
    a, b = (rng.uniform(-9, 9, size).astype(np.float32) for _ in range(2))
    ta, tb = tensor(a, offset), tensor(b, offset)
    assert same(F.relu(ta), oracle.relu(a))
    assert same(F.add2(ta, tb), oracle.add2(a, b))
    assert same(F.relu_backward(ta, tb), oracle.relu_backward(a, b))
    assert same(F.add2_backward(tb), oracle.add2_backward(b))
    assert same(F.fixed_point_quantize(ta, True, 8, 2.0 ** -4), oracle.fixed_point_quantize(a, True, 8, 2.0 ** -4))
    assert same(F.fixed_point_quantize_backward(ta, tb, True, 8, 2.0 ** -4),
                oracle.fixed_point_quantize_backward(a, b, True, 8, 2.0 ** -4))
    if size <= 4096 or size == FEW + 5:
        acc = tensor(a, offset)
        assert same(F.relu_backward(ta, tb, accum=True, dx=acc), oracle.relu_backward(a, b, True, a.copy()))


# planes of one and several chunks of 1024 vectors, the last one ragged, and more than 64 chunks of them (a second round)
@pytest.mark.parametrize("shape", [(3, 5, 64, 64), (2, 3, 64, 65), (2, 2, 100, 124), (1, 2, 516, 1024)])
def test_batch_normalization_chunks(F, shape):
    rng = np.random.RandomState(shape[-1])
    x = rng.randn(*shape).astype(np.float32)
    beta, gamma, mean = (rng.randn(1, shape[1], 1, 1).astype(np.float32) for _ in range(3))
    var = (rng.rand(1, shape[1], 1, 1) + 0.1).astype(np.float32)
    dev = [torch.from_numpy(v).cuda() for v in (x, beta, gamma, mean, var)]
    y = F.batch_normalization(*dev, [1], 0.9, 1e-5, False)
    want = oracle.batch_norm_inference(x.reshape(shape[0], shape[1], -1), beta, gamma, mean, var, 1e-5)
    assert same(y, want)


# two vectors a thread up to 148 * 8 * 256 * 8 of them, four above; and every kind of magnitude of Pow2Quantize: all exponents,
# mantissas around the cut at sqrt(2), zeros of both signs, denormals, infinities, NaN
@pytest.mark.parametrize("form", [(True, True, 8, 1), (True, False, 4, 0), (False, True, 5, 2), (False, False, 3, -3)])
@pytest.mark.parametrize("size", [FEW + 4, 4 * 148 * 8 * 256 * 8 - 1, 4 * 148 * 8 * 256 * 8 + 4 * 1024 + 3])
def test_quantizers_two_and_four_vectors(F, size, form):
    rng = np.random.RandomState(size % 1000)
    a = rng.uniform(-9, 9, size).astype(np.float32)
    cut = np.float32(np.sqrt(2.0)).view(np.int32) & 0x7fffff
    exponents = np.arange(256, dtype=np.int64)[:, None] << 23
    mantissas = np.concatenate([cut + np.arange(-40, 41), [0, 1, 2, 0x400000, 0x7ffffe, 0x7fffff]])[None, :]
    special = (exponents | mantissas).astype(np.uint32).reshape(-1).view(np.float32)
    special = np.concatenate([special, -special])
    a[:special.size] = special
    a[-special.size:] = special[::-1]
    got, want = F.pow2_quantize(tensor(a), *form).cpu().numpy(), oracle.pow2_quantize(a, *form)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan) and np.array_equal(bits(got)[~nan], bits(want)[~nan])
    b = rng.uniform(-9, 9, size).astype(np.float32)
    assert same(F.fixed_point_quantize(tensor(b), True, 8, 2.0 ** -4), oracle.fixed_point_quantize(b, True, 8, 2.0 ** -4))


# small planes, two samples per warp and one: odd numbers of samples, the largest planes of each form, groups of four planes
# that are one sample's and that are not
@pytest.mark.parametrize("shape", [(19, 256, 14, 14), (9, 512, 4, 9), (5, 1000, 16, 16), (5, 1000, 10, 26), (41, 516, 7, 7),
                                   (41, 515, 7, 7), (40, 515, 5, 7), (11, 1024, 31, 33), (3, 8, 14, 14), (1, 4, 7, 7)])
def test_batch_normalization_small_planes(F, shape):
    test_batch_normalization_chunks(F, shape)


# a thread per map (fewer than 24 values, but not 16); values of a map in one run of 64, in several and in parts of one; maps that fill a block of 64 and that do not
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (9, 31, 1, 23), (4, 17, 4, 4), (4, 16, 6, 4), (3, 21, 7, 7), (2, 32, 8, 8), (5, 13, 5, 13), (1, 129, 11, 19), (2, 3, 56, 56)])
def test_global_average_pooling(F, shape):
    x = np.random.RandomState(shape[1]).randn(*shape).astype(np.float32)
    assert same(F.global_average_pooling(tensor(x.reshape(-1)).reshape(shape)), oracle.global_average_pooling(x))


def test_streaming_results(F):
    """Past 240 MB results leave with the streaming policy: the same values."""
    n = (240 << 20) // 4 + 4099
    x = torch.randn(n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    assert torch.equal(F.relu(x), torch.clamp_min(x, 0.0))
    assert torch.equal(F.add2_backward(x), x)
    # the half is added in double precision, as the reference does: in fp32 a value just below a tie would round up
    q = (torch.floor(x.abs().double() * 16.0 + 0.5).clamp_max(127.0) / 16.0).float()
    assert torch.equal(F.fixed_point_quantize(x, True, 8, 2.0 ** -4), torch.where(x < 0, -q, q))
