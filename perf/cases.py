"""The performance cases of this framework: work that its users have it do, through its public entry points.

Six kinds, each in the range of sizes that networks use it at:

  resnet18    a whole binary-weight ResNet-18 forward pass (nnabla_b200.resnet18): the graph as written, with int8
              codes between its layers, or with BatchNormalization folded in; replayed from a CUDA graph or called
              from Python; one image to a batch of 256
  block       one training step of a binary-weight residual block on fixed-point activations: forward with batch
              statistics, then every gradient
  convolution a binary-weight or binary-connect convolution of fp32 activations, alone or with its gradients
  affine      a binary-weight or binary-connect affine layer of fp32 activations, alone or with its gradients
  fixed_point FixedPointQuantize of the activations and of the weights, then the affine of the two
  quantizer   FixedPointQuantize, Pow2Quantize or MinMaxQuantize of a tensor, alone or with its gradient

All data is synthetic and made from the seed.
"""
import math

import torch

from nnabla_b200 import functions as F
from nnabla_b200 import graphs, resnet18

DELTA = 2.0 ** -4  # step of the fixed-point activations, as in the network


def listed():
    return [
        # the network's throughput form: the graph as written, a full batch, replayed
        dict(name="network_as_written_256", kind="resnet18", form="as_written", replay=True, batch=256, size=224),
        # serving: the converted network, a batch collected from requests, replayed
        dict(name="network_folded_64", kind="resnet18", form="folded", replay=True, batch=64, size=224),
        # serving: one image, called function by function from Python
        dict(name="network_folded_1", kind="resnet18", form="folded", replay=False, batch=1, size=224),
        # training: a block of the network's first stage
        dict(name="block_64_56x56", kind="block", batch=128, cin=64, maps=64, size=56, stride=1),
        # training: a block that halves the image and has a projection; a ragged batch and an odd image
        dict(name="block_stride2_27x27", kind="block", batch=20, cin=128, maps=256, size=27, stride=2),
        # a wide 3 x 3 layer on activations that are not quantized
        dict(name="convolution_256_28x28", kind="convolution", train=False, connect=False, batch=128, cin=256,
             maps=256, height=28, width=28, kernel=3, stride=1, group=1),
        # the same kind of layer being trained; channels and image of no round size
        dict(name="convolution_train_ragged", kind="convolution", train=True, connect=True, batch=24, cin=96, maps=160,
             height=35, width=29, kernel=3, stride=1, group=1),
        # a fully connected layer at inference
        dict(name="affine_256x1024x4096", kind="affine", train=False, connect=False, rows=256, inmaps=1024,
             outmaps=4096),
        # a small fully connected layer being trained
        dict(name="affine_train_100x784x500", kind="affine", train=True, connect=False, rows=100, inmaps=784,
             outmaps=500),
        # a large 8-bit affine: both operands quantized, then contracted
        dict(name="fixed_point_8192x4096x8192", kind="fixed_point", rows=8192, inmaps=4096, outmaps=8192),
        # quantizing a large activation in training
        dict(name="quantizer_fixed_point_2p26", kind="quantizer", op="fixed_point", train=True, batch=64, channels=256,
             inner=4096, per_channel=False, observe=False),
        # range-tracking quantization of a small activation in training
        dict(name="quantizer_min_max_small", kind="quantizer", op="min_max", train=True, batch=16, channels=24,
             inner=49, per_channel=True, observe=True),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("resnet18", "block", "convolution", "affine", "fixed_point", "quantizer"))
    while True:
        case = _draw(rng, kind)
        if case is not None:
            return case


def _draw(rng, kind):
    """One case of `kind`, or None where it would cost more than the listed ones or has an empty result."""
    if kind == "resnet18":
        case = dict(kind=kind, form=rng.choice(("as_written", "codes", "folded")), replay=rng.random() < 0.6,
                    batch=_log_int(rng, 1, 256), size=rng.randint(96, 256))
        return case if case["batch"] * case["size"] ** 2 <= 256 * 224 ** 2 else None
    if kind == "block":
        stride = rng.choice((1, 2))
        cin = _log_int(rng, 16, 256)
        case = dict(kind=kind, batch=_log_int(rng, 2, 256), cin=cin, maps=cin * stride, size=rng.randint(7, 64),
                    stride=stride)
        values = case["batch"] * cin * case["size"] ** 2
        return case if values <= 128 * 64 * 56 ** 2 and values * case["maps"] <= 128 * 64 * 64 * 56 ** 2 else None
    if kind == "convolution":
        group = rng.choice((1, 1, 1, 2))
        case = dict(kind=kind, train=rng.random() < 0.5, connect=rng.random() < 0.5, batch=_log_int(rng, 1, 128),
                    cin=group * _log_int(rng, 16, 384), maps=group * _log_int(rng, 16, 384),
                    height=rng.randint(7, 64), width=rng.randint(7, 64), kernel=rng.choice((1, 3, 3, 3, 5)),
                    stride=rng.choice((1, 1, 2)), group=group)
        bound = 1.2e11 / (3 if case["train"] else 1)
        small = case["batch"] * case["cin"] * case["height"] * case["width"] <= 128 * 256 * 28 ** 2
        return case if small and _convolution_flops(case) <= bound else None
    if kind == "affine":
        case = dict(kind=kind, train=rng.random() < 0.5, connect=rng.random() < 0.5, rows=_log_int(rng, 1, 4096),
                    inmaps=_log_int(rng, 32, 8192), outmaps=_log_int(rng, 10, 8192))
        return case if case["rows"] * case["inmaps"] * case["outmaps"] <= 1 << 34 else None
    if kind == "fixed_point":
        case = dict(kind=kind, rows=_log_int(rng, 1, 8192), inmaps=_log_int(rng, 32, 8192),
                    outmaps=_log_int(rng, 10, 8192))
        return case if case["rows"] * case["inmaps"] * case["outmaps"] <= 1 << 38 else None
    op = rng.choice(("fixed_point", "pow2", "min_max"))
    values = _log_int(rng, 1 << 10, 1 << 26)
    channels, inner = _log_int(rng, 1, 256), _log_int(rng, 1, 4096)
    return dict(kind=kind, op=op, train=rng.random() < 0.5, batch=max(1, values // (channels * inner)),
                channels=channels, inner=inner, per_channel=op == "min_max" and rng.random() < 0.5,
                observe=op == "min_max" and rng.random() < 0.5)


def _convolution_out(case):
    pad = case["kernel"] // 2
    return [(case[n] + 2 * pad - case["kernel"]) // case["stride"] + 1 for n in ("height", "width")]


def _convolution_flops(case):
    oh, ow = _convolution_out(case)
    return 2.0 * case["batch"] * case["maps"] * oh * ow * (case["cin"] // case["group"]) * case["kernel"] ** 2


class _Data:
    """Seeded random tensors on the GPU."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, scale=1.0):
        return torch.randn(*shape, device="cuda", generator=self.generator).mul_(scale)

    def uniform(self, low, high, *shape):
        return torch.rand(*shape, device="cuda", generator=self.generator).mul_(high - low).add_(low)


def _weights(data, maps, cin, kernel):
    return data.normal(maps, cin, kernel, kernel, scale=math.sqrt(2.0 / (cin * kernel * kernel)))


def _bn(data, channels):
    shape = (1, channels, 1, 1)
    return dict(beta=data.normal(*shape, scale=0.1), gamma=data.normal(*shape, scale=0.1).add_(1.0),
                mean=data.normal(*shape, scale=0.1), var=data.uniform(0.5, 1.5, *shape))


def _network_parameters(data):
    p = {"stem/conv/W": _weights(data, 64, 3, 7)}

    def bn(name, channels):
        for key, value in _bn(data, channels).items():
            p["%s/%s" % (name, key)] = value.reshape(-1)
    bn("stem/bn", 64)
    for name, cin, maps, stride, projected in resnet18.folded_layers():
        p[name + "/conv1/W"] = _weights(data, maps, cin, 3)
        p[name + "/conv2/W"] = _weights(data, maps, maps, 3)
        bn(name + "/bn1", maps)
        bn(name + "/bn2", maps)
        if projected:
            p[name + "/shortcut/W"] = _weights(data, maps, cin, 1)
            bn(name + "/bn_s", maps)
    p["head/W"] = data.normal(512, 1000, scale=math.sqrt(1.0 / 512))
    p["head/b"] = data.normal(1000, scale=0.01)
    return p


def prepare(case, seed):
    data = _Data(seed)
    return _PREPARE[case["kind"]](case, data)


def run(state):
    return _RUN[state["kind"]](state)


# ---- resnet18 -----------------------------------------------------------------------------------------------------

def _prepare_resnet18(case, data):
    params = _network_parameters(data)
    images = data.normal(case["batch"], 3, case["size"], case["size"])

    def zeros_like(t, shape=None):
        return torch.zeros(tuple(t.shape) if shape is None else shape, device="cuda")
    if case["form"] == "as_written":
        network = resnet18.Runner(F, params, zeros_like, codes_sideband=True)
    elif case["form"] == "codes":
        network = resnet18.Runner(F, params, zeros_like, fused="codes", prepared_weights=True)
    else:
        network = resnet18.FoldedRunner(F, params)
    state = dict(kind="resnet18", network=network, call=network, images=images)
    if case["replay"]:
        state["call"] = graphs.Captured(network, images)
        state["images"] = state["call"].static_inputs[0]  # where such a program puts its images
    return state


def _run_resnet18(s):
    logits = s["call"](s["images"])
    binary = getattr(s["network"], "side", {})  # the graph as written binarises its weights in every pass
    return dict(logits=logits, binary={name: list(pair) for name, pair in binary.items()})


# ---- block --------------------------------------------------------------------------------------------------------

def _prepare_block(case, data):
    batch, cin, maps, size, stride = (case[k] for k in ("batch", "cin", "maps", "size", "stride"))
    out = (size - 1) // stride + 1
    s = dict(kind="block", stride=stride, x=data.normal(batch, cin, size, size).relu_(),
             dy=data.normal(batch, maps, out, out, scale=1e-2), layers={})
    layers = [("conv1", cin, 3), ("conv2", maps, 3)] + ([("shortcut", cin, 1)] if stride != 1 else [])
    for name, channels, kernel in layers:
        w = _weights(data, maps, channels, kernel)
        s["layers"][name] = dict(w=w, wb=torch.zeros_like(w), alpha=torch.zeros(maps, device="cuda"),
                                 pad=(kernel // 2,) * 2, stride=(1, 1) if name == "conv2" else (stride, stride),
                                 bn=_bn(data, maps))
    return s


def _forward_layer(layer, x):
    layer["x"] = x
    layer["r"] = F.binary_weight_convolution(x, layer["w"], layer["wb"], layer["alpha"], None, 1, layer["pad"],
                                             layer["stride"], fixed_point_delta=DELTA)
    bn = layer["bn"]
    y, layer["mean"], layer["var"] = F.batch_normalization(layer["r"], bn["beta"], bn["gamma"], bn["mean"], bn["var"],
                                                           [1], 0.9, 1e-5, True, output_stat=True)
    return y


def _backward_layer(layer, dy, dx=None):
    """Gradients of one convolution and its BatchNormalization; dx: the gradient to add the input's to."""
    dr, dbeta, dgamma = F.batch_normalization_backward(layer["r"], dy, layer["bn"]["gamma"], layer["mean"],
                                                       layer["var"])
    dx, dw, _ = F.binary_weight_convolution_backward(
        layer["x"], layer["wb"], layer["alpha"], dr, 1, layer["pad"], layer["stride"],
        propagate_down=(True, True, False), accum=(dx is not None, False, False), grads=(dx, None, None),
        fixed_point_delta=DELTA)
    return dx, [dw, dbeta, dgamma]


def _run_block(s):
    layers = s["layers"]
    h = F.fixed_point_quantize(s["x"], True, 8, DELTA)
    a = F.relu(_forward_layer(layers["conv1"], h))
    q = F.fixed_point_quantize(a, True, 8, DELTA)
    r = _forward_layer(layers["conv2"], q)
    shortcut = _forward_layer(layers["shortcut"], h) if "shortcut" in layers else h
    y = F.relu(F.add2(r, shortcut))

    gradients = {}
    dsum = F.relu_backward(y, s["dy"])
    dq, gradients["conv2"] = _backward_layer(layers["conv2"], dsum)
    da = F.fixed_point_quantize_backward(a, dq, True, 8, DELTA)
    dr = F.relu_backward(a, da)
    if "shortcut" in layers:
        dh, gradients["shortcut"] = _backward_layer(layers["shortcut"], dsum)
    else:
        dh = F.add2_backward(dsum)
    dh, gradients["conv1"] = _backward_layer(layers["conv1"], dr, dh)
    dx = F.fixed_point_quantize_backward(s["x"], dh, True, 8, DELTA)
    updated = {name: [layer[k] for k in ("wb", "alpha", "mean", "var")] + [layer["bn"]["mean"], layer["bn"]["var"]]
               for name, layer in layers.items()}
    return dict(y=y, dx=dx, gradients=gradients, updated=updated)


# ---- convolution and affine ---------------------------------------------------------------------------------------

def _prepare_convolution(case, data):
    shape = (case["batch"], case["cin"], case["height"], case["width"])
    w = _weights(data, case["maps"], case["cin"] // case["group"], case["kernel"])
    geometry = dict(pad=(case["kernel"] // 2,) * 2, stride=(case["stride"],) * 2, group=case["group"])
    s = dict(kind="convolution", connect=case["connect"], geometry=geometry, x=data.normal(*shape).relu_(), w=w,
             wb=torch.zeros_like(w), alpha=torch.zeros(case["maps"], device="cuda"),
             b=data.normal(case["maps"], scale=0.01))
    if case["train"]:
        s["dy"] = data.normal(case["batch"], case["maps"], *_convolution_out(case), scale=1e-2)
    return s


def _run_convolution(s):
    g = s["geometry"]
    if s["connect"]:
        out = [F.binary_connect_convolution(s["x"], s["w"], s["wb"], s["b"], **g), s["wb"]]
        if "dy" in s:
            out += F.binary_connect_convolution_backward(s["x"], s["wb"], s["dy"], **g)
    else:
        out = [F.binary_weight_convolution(s["x"], s["w"], s["wb"], s["alpha"], s["b"], **g), s["wb"], s["alpha"]]
        if "dy" in s:
            out += F.binary_weight_convolution_backward(s["x"], s["wb"], s["alpha"], s["dy"], **g)
    return out


def _prepare_affine(case, data):
    rows, inmaps, outmaps = case["rows"], case["inmaps"], case["outmaps"]
    w = data.normal(inmaps, outmaps, scale=0.02)
    s = dict(kind="affine", connect=case["connect"], x=data.normal(rows, inmaps), w=w, wb=torch.zeros_like(w),
             alpha=torch.zeros(outmaps, device="cuda"), b=data.normal(outmaps, scale=0.01))
    if case["train"]:
        s["dy"] = data.normal(rows, outmaps, scale=1e-2)
    return s


def _run_affine(s):
    if s["connect"]:
        out = [F.binary_connect_affine(s["x"], s["w"], s["wb"], s["b"]), s["wb"]]
        if "dy" in s:
            out += F.binary_connect_affine_backward(s["x"], s["wb"], s["dy"])
    else:
        out = [F.binary_weight_affine(s["x"], s["w"], s["wb"], s["alpha"], s["b"]), s["wb"], s["alpha"]]
        if "dy" in s:
            out += F.binary_weight_affine_backward(s["x"], s["wb"], s["alpha"], s["dy"])
    return out


# ---- fixed_point --------------------------------------------------------------------------------------------------

def _prepare_fixed_point(case, data):
    return dict(kind="fixed_point", x=data.normal(case["rows"], case["inmaps"]),
                w=data.normal(case["inmaps"], case["outmaps"], scale=0.02), b=data.normal(case["outmaps"], scale=0.01))


def _run_fixed_point(s):
    delta_x, delta_w = 2.0 ** -5, 2.0 ** -10
    xq = F.fixed_point_quantize(s["x"], True, 8, delta_x)
    wq = F.fixed_point_quantize(s["w"], True, 8, delta_w)
    return [F.affine(xq, wq, s["b"], fixed_point=(delta_x, delta_w)), xq, wq]


# ---- quantizer ----------------------------------------------------------------------------------------------------

def _prepare_quantizer(case, data):
    shape = (case["batch"], case["channels"], case["inner"])
    s = dict(kind="quantizer", op=case["op"], observe=case["observe"], x=data.uniform(-4.5, 4.5, *shape))
    if case["op"] == "min_max":
        q = (1, case["channels"] if case["per_channel"] else 1, 1)
        s["ranges"] = [torch.full(q, v, device="cuda") for v in (-4.0, 4.0, 0.0, 255.0)]
    if case["train"]:
        s["dy"] = data.normal(*shape)
    return s


def _run_quantizer(s):
    x, dy = s["x"], s.get("dy")
    if s["op"] == "fixed_point":
        out = [F.fixed_point_quantize(x, True, 8, DELTA)]
        if dy is not None:
            out.append(F.fixed_point_quantize_backward(x, dy, True, 8, DELTA))
    elif s["op"] == "pow2":
        out = [F.pow2_quantize(x, True, True, 8, 1)]
        if dy is not None:
            out.append(F.pow2_quantize_backward(x, dy, True, True, 8, 1))
    else:
        observe = dict(x_min_max=s["observe"], ema=s["observe"])
        out = [F.min_max_quantize(x, *s["ranges"], **observe)] + s["ranges"][:2]
        if dy is not None:
            out += F.min_max_quantize_backward(x, *s["ranges"], dy, **observe)
    return out


_PREPARE = dict(resnet18=_prepare_resnet18, block=_prepare_block, convolution=_prepare_convolution,
                affine=_prepare_affine, fixed_point=_prepare_fixed_point, quantizer=_prepare_quantizer)
_RUN = dict(resnet18=_run_resnet18, block=_run_block, convolution=_run_convolution, affine=_run_affine,
            fixed_point=_run_fixed_point, quantizer=_run_quantizer)


def work(case):
    """Bytes and operations of one pass that no implementation can do without: inputs read once, outputs written once."""
    kind = case["kind"]
    if kind == "resnet18":
        weights = sum(maps * cin * 9 + maps * maps * 9 + (maps * cin if projected else 0)
                      for _, cin, maps, _, projected in resnet18.folded_layers())
        other = 64 * 3 * 49 + 512 * 1000 + 1000
        values = case["batch"] * (3 * case["size"] ** 2 + 1000) + other
        # as written: float weights in, binary weights out; the other forms hold one byte for each
        total = 4.0 * values + (8.0 if case["form"] == "as_written" else 1.0) * weights
        return dict(bytes=total, flops=2.0 * case["batch"] * resnet18.conv_macs_per_image(case["size"], case["size"]))
    if kind == "block":
        out = (case["size"] - 1) // case["stride"] + 1
        pixels = case["batch"] * out * out
        weights = case["maps"] * (9 * case["cin"] + 9 * case["maps"] + (case["cin"] if case["stride"] != 1 else 0))
        x, y = case["batch"] * case["cin"] * case["size"] ** 2, pixels * case["maps"]
        # x and dy in, y and dx out; float weights in, binary weights and gradients out
        return dict(bytes=4.0 * (2 * x + 2 * y + 3 * weights), flops=6.0 * pixels * weights)
    if kind == "convolution":
        oh, ow = _convolution_out(case)
        x = case["batch"] * case["cin"] * case["height"] * case["width"]
        y = case["batch"] * case["maps"] * oh * ow
        weights = case["maps"] * (case["cin"] // case["group"]) * case["kernel"] ** 2
        times = 2 if case["train"] else 1
        return dict(bytes=4.0 * (times * (x + y) + (1 + times) * weights),
                    flops=(3 if case["train"] else 1) * _convolution_flops(case))
    if kind in ("affine", "fixed_point"):
        rows, inmaps, outmaps = case["rows"], case["inmaps"], case["outmaps"]
        x, y, weights = rows * inmaps, rows * outmaps, inmaps * outmaps
        if kind == "fixed_point":
            return dict(bytes=4.0 * (2 * x + 2 * weights + y + outmaps), flops=2.0 * rows * weights)
        times = 2 if case["train"] else 1
        return dict(bytes=4.0 * (times * (x + y) + (1 + times) * weights + times * outmaps),
                    flops=(6.0 if case["train"] else 2.0) * rows * weights)
    values = case["batch"] * case["channels"] * case["inner"]
    return dict(bytes=4.0 * values * (4 if case["train"] else 2), flops=1.0 * values * (2 if case["train"] else 1))


def tolerance(case):
    kind = case["kind"]
    if kind == "resnet18":
        # activations of 8 bits: a rounding of the stem's fp32 sums can move a value by one step, which the layers
        # behind it carry into the logits
        return dict(rel=5e-3, max=5e-2)
    if kind == "block":
        # an 8-bit step of the hidden activation can turn over where the batch statistics round differently
        return dict(rel=1e-4, max=0.2)
    if kind in ("convolution", "affine"):
        return dict(rel=1e-5, max=4e-4)
    if kind == "fixed_point":
        return dict(rel=1e-6, max=4e-5)
    # one rounding each; a range gradient is an fp32 sum
    return dict(rel=1e-5, max=4e-4) if case["op"] == "min_max" and case["train"] else "exact"
