"""int8 convolutions with several column tiles of 32 or 64 maps, a block each (few pixels, many maps): stride 1 with one
box of pixels for all taps, stride 2 and 1 x 1 with a box per tap; ragged maps and images, with the residual as codes or
fp32, against 64-bit sums: codes and fp32 results exactly."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# batch, channels, maps, height, width, kernel, stride
CASES = [(1, 512, 512, 7, 7, 3, 1), (3, 512, 500, 7, 5, 3, 1), (1, 256, 256, 14, 14, 3, 1), (9, 256, 130, 14, 13, 3, 1),
         (2, 128, 128, 28, 28, 3, 1), (1, 96, 72, 9, 30, 3, 1), (5, 200, 300, 8, 8, 5, 1), (16, 256, 256, 14, 14, 3, 1),
         (1, 256, 512, 14, 14, 3, 2), (2, 256, 512, 14, 14, 1, 2), (1, 128, 200, 28, 27, 3, 2), (20, 256, 256, 14, 14, 3, 1)]


@pytest.mark.parametrize("batch,channels,maps,height,width,kernel,stride", CASES)
@pytest.mark.parametrize("form", ["residual", "float", "plain"])
def test_few_pixels_many_maps(batch, channels, maps, height, width, kernel, stride, form):
    from nnabla_b200 import functions as F
    rng = np.random.RandomState(maps + width)
    dev = lambda a: torch.from_numpy(a).cuda()
    prep = F.prepare_binary_weights(dev(rng.randn(maps, channels, kernel, kernel).astype(np.float32)))
    scale, bias = dev((0.002 + 0.002 * rng.rand(maps)).astype(np.float32)), dev(rng.randn(maps).astype(np.float32))
    pad = kernel // 2
    out_h, out_w = (height + 2 * pad - kernel) // stride + 1, (width + 2 * pad - kernel) // stride + 1
    codes = torch.zeros(batch, height * width, F.codes_nhwc_slots(channels), dtype=torch.int8, device="cuda")
    codes[:, :, :channels] = dev(rng.randint(0, 128, (batch, height * width, channels)).astype(np.int8))
    slots = F.codes_nhwc_slots(maps)
    res = torch.zeros(batch, out_h * out_w, slots, dtype=torch.int8, device="cuda")
    res[:, :, :maps] = dev(rng.randint(-127, 128, (batch, out_h * out_w, maps)).astype(np.int8))
    kw = dict(residual=dict(residual_codes=res, residual_delta=2.0 ** -5), float=dict(relu=False, output="float"),
              plain=dict())[form]
    y, shape = F.convolution_codes_folded(codes, (batch, channels, height, width), prep, scale, bias, (pad, pad),
                                          (stride, stride), delta=2.0 ** -4, **kw)
    F.check_device_status()
    planes = lambda t, c: t[:, :, :c].double().transpose(1, 2).reshape(batch, c, -1)
    x = planes(codes, channels).reshape(batch, channels, height, width)
    acc = torch.nn.functional.conv2d(x, prep.binary_weight.double(), padding=pad, stride=stride).reshape(batch, maps, -1)
    v = (acc * scale.double().view(1, -1, 1) + bias.double().view(1, -1, 1)).float()
    if form == "residual":
        v = (planes(res, maps) * 2.0 ** -5 + v.double()).float()
    assert shape == (batch, maps, out_h, out_w) and not y[:, :, maps:].any()
    if form == "float":
        assert torch.equal(planes(y, maps).float(), v)
    else:
        want = torch.floor(v.clamp(min=0).double() * 16 + 0.5).clamp(max=127)
        assert torch.equal(planes(y, maps), want)
