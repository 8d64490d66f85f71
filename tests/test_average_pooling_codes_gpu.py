"""GlobalAveragePooling of codes: integer sums (steps that are powers of two) against the sequential sums of the plain
function on the fp32 values, bit for bit, at the edges of its 512-slot blocks and 8 pixel shares."""
import numpy as np
import pytest
import torch

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 512, 7, 7), (3, 20, 1, 1), (2, 513, 2, 4), (5, 64, 3, 3), (2, 1000, 5, 13)])
@pytest.mark.parametrize("delta", [2.0 ** -4, 2.0 ** -90, 2.0 ** 101, 0.1])
def test_global_average_pooling_of_codes(shape, delta):
    from nnabla_b200 import functions as F
    N, C, H, W = shape
    k = np.random.RandomState(C).randint(-127, 128, shape)
    codes = torch.zeros(N, H * W, F.codes_nhwc_slots(C, 1), dtype=torch.int8)
    codes[:, :, :C] = torch.from_numpy(k.reshape(N, C, H * W).transpose(0, 2, 1).astype(np.int8))
    y = F.global_average_pooling_codes(codes.cuda(), shape, delta)
    x = (k.astype(np.float32) * np.float32(delta)).astype(np.float32)
    want = oracle.global_average_pooling(x)
    assert np.array_equal(y.cpu().numpy().reshape(-1), want.reshape(-1))
