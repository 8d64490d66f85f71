"""The quantizer with channel-last codes against the plain quantizer and the oracle, bit for bit, on the values where
rounding and limits decide: every tie and limit of the grid with its neighbours, zeros of both signs, denormals,
infinities; planes and channels at the edges of its 128-pixel, 64-channel blocks; steps at the ends of their range."""
import numpy as np
import pytest
import torch

from golden_util import bits
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    from nnabla_b200 import _capi, functions
    _capi.call("nb200_check_device")
    return functions


def special_values(n, sign, delta):
    top = 2 ** (n - sign)
    grid = (np.arange(-2 * top - 4, 2 * top + 5) * np.float64(delta) / 2).astype(np.float32)
    v = np.concatenate([grid, np.nextafter(grid, np.float32(np.inf)), np.nextafter(grid, np.float32(-np.inf))])
    tiny = np.array([0.0, -0.0, 1e-45, -1e-45, 1.2e-38, -1.2e-38, 3e38, -3e38, np.inf, -np.inf], np.float32)
    return np.concatenate([tiny, v])


@pytest.mark.parametrize("shape", [(1, 1, 2, 2), (2, 63, 4, 31), (1, 64, 8, 16), (2, 65, 4, 33), (3, 130, 12, 11)])
@pytest.mark.parametrize("n,sign,delta", [(8, True, 2.0 ** -4), (7, False, 2.0 ** -3), (2, True, 1.0), (8, True, 0.1),
                                          (8, True, 2.0 ** 110), (8, True, 2.0 ** -119)])
def test_codes_at_the_edges(F, shape, n, sign, delta):
    L = F.L
    N, C, H, W = shape
    rng = np.random.RandomState(n + C)
    with np.errstate(over="ignore", invalid="ignore"):
        pool = special_values(n, sign, delta)
        x = np.concatenate([pool, (rng.randn(N * C * H * W) * delta * 2 ** (n - 1)).astype(np.float32)])
    x = (x[:N * C * H * W] if C > 1 else rng.permutation(pool)[:N * C * H * W]).reshape(shape)
    gx = torch.from_numpy(x).cuda()
    y = torch.empty_like(gx)
    codes = torch.empty(N, H * W, F.codes_nhwc_slots(C, 1), dtype=torch.int8, device="cuda")
    L.nb200_fixed_point_quantize_nhwc_codes_f32(gx, y, codes, N, C, H * W, sign, n, delta)
    want = oracle.fixed_point_quantize(x, sign, n, delta)
    assert np.array_equal(bits(y.cpu().numpy()), bits(want))
    assert np.array_equal(bits(y.cpu().numpy()), bits(F.fixed_point_quantize(gx, sign, n, delta).cpu().numpy()))
    k = np.rint(want.astype(np.float64) / np.float64(np.float32(delta))).astype(np.int8)
    got = codes.cpu().numpy()
    assert np.array_equal(got[:, :, :C], k.reshape(N, C, H * W).transpose(0, 2, 1)) and not got[:, :, C:].any()


def test_a_nan_stays(F):
    L = F.L
    x = torch.full((1, 4, 2, 2), float("nan"), device="cuda")
    x[0, 0] = 1.0
    y, codes = torch.empty_like(x), torch.empty(1, 4, 64, dtype=torch.int8, device="cuda")
    L.nb200_fixed_point_quantize_nhwc_codes_f32(x, y, codes, 1, 4, 4, True, 8, 2.0 ** -4)
    assert torch.equal(torch.isnan(y), torch.isnan(x)) and torch.equal(y[0, 0], x[0, 0])
