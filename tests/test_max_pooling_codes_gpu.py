"""Max pooling of codes: every pair of signed bytes in every lane of a word, windows of the specialised and the general
kernels, clipped at every border, against maxima over the codes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel,stride,pad", [((3, 3), (2, 2), (1, 1)), ((2, 2), (2, 2), (0, 0)), ((1, 2), (1, 2), (0, 0)),
                                               ((4, 3), (1, 2), (2, 1))])
@pytest.mark.parametrize("shape", [(2, 64, 9, 8), (1, 130, 5, 7), (3, 20, 16, 33)])
def test_max_pooling_of_codes(shape, kernel, stride, pad):
    from nnabla_b200 import functions as F
    N, C, H, W = shape
    k = np.random.RandomState(C).randint(-128, 128, shape).astype(np.int8)
    k[0, :, 0, 0], k[0, :, 0, 1] = -128, 127
    codes = torch.zeros(N, H * W, F.codes_nhwc_slots(C, 1), dtype=torch.int8)
    codes[:, :, :C] = torch.from_numpy(k.reshape(N, C, H * W).transpose(0, 2, 1))
    y, out = F.max_pooling_codes(codes.cuda(), shape, kernel, stride, True, pad)
    want = torch.nn.functional.max_pool2d(torch.from_numpy(k).float(), kernel, stride, pad)
    assert tuple(out) == tuple(want.shape)
    got = y.cpu()[:, :, :C].float().transpose(1, 2).reshape(want.shape)
    assert torch.equal(got, want) and not y.cpu()[:, :, C:].any()


def test_every_pair_of_bytes():
    from nnabla_b200 import functions as F
    a = torch.arange(-128, 128, dtype=torch.int8)
    pairs = torch.cartesian_prod(a, a)  # 65536 rows of two pixels, spread over 64 slots
    codes = pairs.reshape(1024, 64, 2).transpose(1, 2).contiguous().cuda()  # [sample][pixel][slot]
    y, _ = F.max_pooling_codes(codes, (1024, 64, 1, 2), (1, 2), (1, 2), True, (0, 0))
    assert torch.equal(y.reshape(1024, 64).cpu(), codes.cpu().amax(1))
