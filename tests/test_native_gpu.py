"""Whole calls of the binding against the mirror's own path: the same bits, and the same errors."""
import pytest
import torch

from nnabla_b200 import functions as F

pytestmark = pytest.mark.gpu


def flat(v):
    return [t for e in v for t in flat(e)] if isinstance(v, (tuple, list)) else [v]


@pytest.fixture
def t():
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x = (r(2, 32, 9, 11) * 8).round().clamp(-127, 127) / 16
    w = r(48, 32, 3, 3)
    return dict(x=x, w=w, wb=torch.empty_like(w), alpha=torch.empty(48, device="cuda"), b=r(48), dy=r(2, 48, 5, 6),
                codes=F.fixed_point_codes_nhwc(x, 1 / 16), prep=F.prepare_binary_weights(w, 1, 1.0), s=r(48).abs(), r=r)


G = dict(pad=(1, 1), stride=(2, 2))
CALLS = {
    "folded_convolution": [
        lambda t: F.convolution_codes_folded(t["codes"], t["x"].shape, t["prep"], t["s"], t["b"], **G),
        lambda t: F.convolution_codes_folded(t["codes"], t["x"].shape, t["prep"], t["s"], **G, relu=False, output="float"),
        lambda t: F.convolution_codes_folded(t["codes"], t["x"].shape, t["prep"], t["s"][:5], t["b"], **G),
        lambda t: F.convolution_codes_folded(t["codes"], t["x"].shape, t["prep"], t["s"], t["b"], **G, output="?"),
    ],
    "binary_convolution": [
        lambda t: F.binary_weight_convolution(t["x"], t["w"], t["wb"], t["alpha"], t["b"], **G, fixed_point_delta=1 / 16),
        lambda t: F.binary_connect_convolution(t["x"], t["w"], t["wb"], **G),
        lambda t: F.binary_connect_convolution(t["x"][:, :16], t["w"], t["wb"], **G),
    ],
    "binary_convolution_backward": [
        lambda t: F.binary_weight_convolution_backward(t["x"], t["wb"].fill_(1), t["s"], t["dy"], **G),
        lambda t: F.binary_connect_convolution_backward(
            t["x"], t["wb"].fill_(1), t["dy"], **G, propagate_down=(True, False, True), accum=(True, False, False),
            grads=(torch.ones_like(t["x"]), None, None)),
        lambda t: F.binary_connect_convolution_backward(t["x"], t["wb"], t["dy"], **G, accum=(True, False, False)),
        lambda t: F.binary_connect_convolution_backward(t["x"], t["wb"], t["dy"][:1], **G),
    ],
    "batch_normalization": [
        lambda t: F.batch_normalization(t["dy"], t["b"], t["s"], t["b"] * 1, t["s"] * 1, output_stat=True),
        lambda t: F.batch_normalization(t["dy"], None, t["s"].view(1, -1, 1, 1), t["b"], t["s"], batch_stat=False),
        lambda t: F.batch_normalization(t["x"], t["b"], t["s"], t["b"], t["s"]),
    ],
    "batch_normalization_backward": [
        lambda t: F.batch_normalization_backward(t["dy"], t["dy"] * 2, t["s"], t["b"], t["s"]),
        lambda t: F.batch_normalization_backward(t["dy"], t["dy"] * 2, None, t["b"], t["s"], batch_stat=False,
                                                 propagate_down=(True, False, True)),
        lambda t: F.batch_normalization_backward(t["dy"], t["dy"], t["s"], t["b"], t["s"], accum=(False, True, False)),
    ],
    "min_max_quantize": [
        lambda t: F.min_max_quantize(t["x"], *ranges(t, 32), x_min_max=True, ema=True),
        lambda t: F.min_max_quantize(t["x"], *ranges(t, 1)),
        lambda t: F.min_max_quantize(t["x"], *ranges(t, 16)),
    ],
    "min_max_quantize_backward": [
        lambda t: F.min_max_quantize_backward(t["x"], *ranges(t, 32), t["x"] * 2, x_min_max=True),
        lambda t: F.min_max_quantize_backward(t["x"], *ranges(t, 1), t["x"] * 2, accum=(True, False, False),
                                              grads=(torch.ones_like(t["x"]), None, None)),
        lambda t: F.min_max_quantize_backward(t["x"], *ranges(t, 1), t["x"] * 2, propagate_down=(False, True, False),
                                              grads=(torch.ones_like(t["x"]), None, None)),
        lambda t: F.min_max_quantize_backward(t["x"], *ranges(t, 1), t["dy"]),
    ],
}


def ranges(t, n):
    return [torch.full((1, n, 1, 1), v, device="cuda") for v in (-1.0, 1.5, 0.0, 255.0)]


@pytest.mark.parametrize("name,k", [(n, k) for n, calls in CALLS.items() for k in range(len(calls))])
def test_same_as_the_full_path(monkeypatch, t, name, k):
    def outcome():
        try:
            return [v.clone() if torch.is_tensor(v) else v for v in flat(CALLS[name][k](t))]
        except Exception as e:
            return type(e), str(e)
    got = outcome()
    monkeypatch.setattr(F.L, name, lambda *a: None)
    want = outcome()
    assert type(got) is type(want) and len(got) == len(want)
    for a, b in zip(got, want):
        assert torch.equal(a, b) if torch.is_tensor(a) else a == b
