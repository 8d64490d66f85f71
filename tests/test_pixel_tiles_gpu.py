"""int8 convolutions whose blocks do several tiles of pixels one after the other, with as many on the way as there is room
for: 1 to 9 tiles per block (fewer and more than the buffers), pairs of row blocks, ragged last rows and images, one and two
blocks of channels, against 64-bit sums: codes and fp32 results exactly."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# batch, channels, maps, height, width, kernel, dilation
CASES = [(12, 64, 64, 56, 56, 3, 1), (37, 64, 64, 56, 56, 3, 1), (64, 50, 60, 49, 56, 3, 1), (95, 64, 40, 55, 53, 3, 1),
         (70, 64, 128, 28, 28, 3, 1), (180, 40, 100, 27, 28, 3, 1), (110, 128, 128, 28, 28, 3, 1), (90, 100, 64, 27, 26, 3, 1),
         (160, 64, 64, 14, 14, 5, 2), (600, 16, 16, 14, 14, 3, 1), (1300, 16, 24, 7, 7, 3, 1)]


@pytest.mark.parametrize("batch,channels,maps,height,width,kernel,dilation", CASES)
@pytest.mark.parametrize("form", ["residual", "float"])
def test_several_tiles_per_block(batch, channels, maps, height, width, kernel, dilation, form):
    from nnabla_b200 import functions as F
    rng = np.random.RandomState(batch + width)
    dev = lambda a: torch.from_numpy(a).cuda()
    prep = F.prepare_binary_weights(dev(rng.randn(maps, channels, kernel, kernel).astype(np.float32)))
    scale, bias = dev((0.002 + 0.002 * rng.rand(maps)).astype(np.float32)), dev(rng.randn(maps).astype(np.float32))
    pad, slots, pixels = dilation * (kernel // 2), F.codes_nhwc_slots(maps), height * width
    torch.manual_seed(batch)
    codes = torch.zeros(batch, pixels, F.codes_nhwc_slots(channels), dtype=torch.int8, device="cuda")
    codes[:, :, :channels] = torch.randint(0, 128, (batch, pixels, channels), device="cuda").to(torch.int8)
    res = torch.zeros(batch, pixels, slots, dtype=torch.int8, device="cuda")
    res[:, :, :maps] = torch.randint(-127, 128, (batch, pixels, maps), device="cuda").to(torch.int8)
    kw = dict(residual_codes=res, residual_delta=2.0 ** -5) if form == "residual" else dict(relu=False, output="float")
    y, shape = F.convolution_codes_folded(codes, (batch, channels, height, width), prep, scale, bias, (pad, pad), (1, 1),
                                          (dilation, dilation), delta=2.0 ** -4, **kw)
    F.check_device_status()
    planes = lambda t, c: t[:, :, :c].double().transpose(1, 2).reshape(batch, c, -1)
    x = planes(codes, channels).reshape(batch, channels, height, width)
    acc = torch.nn.functional.conv2d(x, prep.binary_weight.double(), padding=pad, dilation=dilation).reshape(batch, maps, -1)
    v = (acc * scale.double().view(1, -1, 1) + bias.double().view(1, -1, 1)).float()
    assert shape == (batch, maps, height, width) and not y[:, :, maps:].any()
    if form == "float":
        assert torch.equal(planes(y, maps).float(), v)
    else:
        v = (planes(res, maps) * 2.0 ** -5 + v.double()).float()
        assert torch.equal(planes(y, maps), torch.floor(v.clamp(min=0).double() * 16 + 0.5).clamp(max=127))


def test_plain_fp32_result():
    from nnabla_b200 import functions as F
    torch.manual_seed(5)
    batch, channels, maps, height, width = 50, 64, 60, 55, 56
    codes = torch.zeros(batch, height * width, F.codes_nhwc_slots(channels), dtype=torch.int8, device="cuda")
    codes[:, :, :channels] = torch.randint(0, 128, (batch, height * width, channels), device="cuda").to(torch.int8)
    w = torch.randn(maps, channels, 3, 3, device="cuda")
    y = F.binary_weight_convolution_from_codes(codes, (batch, channels, height, width), w, torch.zeros_like(w), None, None,
                                               (1, 1), (1, 1), activation_delta=2.0 ** -4)
    F.check_device_status()
    x = codes[:, :, :channels].double().transpose(1, 2).reshape(batch, channels, height, width)
    acc = torch.nn.functional.conv2d(x, torch.where(w > 0, 1.0, -1.0).double(), padding=1)
    assert torch.equal(y.double(), acc * 2.0 ** -4)
