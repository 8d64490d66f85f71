"""A graph of folded convolutions in one call against the same calls one by one, bit for bit: sources and residuals that
are the input, codes or fp32 results, used once, twice or much later; forms that the binding hands back to Python."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    from nnabla_b200 import functions
    return functions


def layer(F, maps, channels, kernel, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(maps, channels, kernel, kernel, device="cuda", generator=g)
    return (F.prepare_binary_weights(w), torch.rand(maps, device="cuda", generator=g) * 0.01 + 0.001,
            torch.randn(maps, device="cuda", generator=g))


def one_by_one(F, codes, shape, steps, delta):
    results = [(codes, shape, True)]
    for source, prep, scale, bias, pad, stride, residual, relu, is_codes in steps:
        added = None if residual is None else results[residual]
        kw = {} if added is None else (dict(residual_codes=added[0], residual_delta=delta) if added[2]
                                       else dict(residual=added[0]))
        y, out = F.convolution_codes_folded(results[source][0], results[source][1], prep, scale, bias, pad, stride,
                                            relu=relu, delta=delta, output="codes" if is_codes else "float", **kw)
        results.append((y, out, is_codes))
    return results[-1][:2]


@pytest.mark.parametrize("batch,size", [(1, 14), (5, 9)])
def test_same_results(F, batch, size):
    one, pad = (1, 1), (1, 1)
    steps = ((0,) + layer(F, 96, 96, 3, 1) + (pad, one, None, True, True),
             (1,) + layer(F, 96, 96, 3, 2) + (pad, one, 0, True, True),       # the input as the residual
             (2,) + layer(F, 160, 96, 3, 3) + (pad, (2, 2), None, True, True),
             (2,) + layer(F, 160, 96, 1, 4) + ((0, 0), (2, 2), None, False, False),
             (3,) + layer(F, 160, 160, 3, 5) + (pad, one, 4, True, True),     # an fp32 residual
             (5,) + layer(F, 160, 160, 3, 6)[:2] + (None, pad, one, 3, True, True),  # no bias; an earlier result
             (6,) + layer(F, 40, 160, 1, 7) + (None, None, None, False, False))
    g = torch.Generator(device="cuda").manual_seed(9)
    codes = torch.randint(0, 128, (batch, size * size, F.codes_nhwc_slots(96)), device="cuda", generator=g, dtype=torch.int8)
    codes[:, :, 96:] = 0
    for last in (1, 5, 6, 7):
        got, shape = F.folded_convolutions(codes, (batch, 96, size, size), steps[:last], 2.0 ** -4)
        want, want_shape = one_by_one(F, codes, (batch, 96, size, size), steps[:last], 2.0 ** -4)
        assert shape == want_shape and torch.equal(got, want)
    # a scale that is not contiguous: the mirror's own loop
    odd = steps[0][:2] + (torch.stack([steps[0][2], steps[0][2]], 1)[:, 0],) + steps[0][3:]
    got, _ = F.folded_convolutions(codes, (batch, 96, size, size), (odd,) + steps[1:3], 2.0 ** -4)
    assert torch.equal(got, one_by_one(F, codes, (batch, 96, size, size), steps[:3], 2.0 ** -4)[0])


def test_wrong_steps_raise(F):
    prep, scale, bias = layer(F, 64, 64, 3, 1)
    codes = torch.zeros(1, 64, 64, dtype=torch.int8, device="cuda")
    good = (0, prep, scale, bias, (1, 1), (1, 1), None, True, True)
    for bad in (good[:2] + (scale[:5],) + good[3:], (0, prep, scale, bias, (0, 0), (1, 1), 0, True, True),
                (4,) + good[1:], (0,) + layer(F, 64, 32, 3, 1) + good[4:]):
        with pytest.raises(Exception):
            F.folded_convolutions(codes, (1, 64, 8, 8), (good, bad), 2.0 ** -4)
    # results that no step before has, counted from the end too: on the fast path and in the mirror's own loop
    for odd in (good, good[:2] + (torch.stack([scale, scale], 1)[:, 0],) + good[3:]):
        for source, residual in ((-1, None), (2, None), (0, -1), (0, 2), (-1, -1)):
            bad = (source,) + good[1:6] + (residual, True, True)
            with pytest.raises(IndexError):
                F.folded_convolutions(codes, (1, 64, 8, 8), (odd, bad), 2.0 ** -4)


def test_network(F):
    from nnabla_b200 import resnet18
    import numpy as np
    p = {k: torch.from_numpy(v).cuda() for k, v in resnet18.init_parameters(np.random.RandomState(3), num_classes=16).items()}
    x = torch.randn(3, 3, 64, 64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    trace = []
    assert torch.equal(resnet18.FoldedRunner(F, p)(x), resnet18.FoldedRunner(F, p, trace)(x))
    assert len(trace) == 21
