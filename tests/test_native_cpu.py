"""The binding's shape arithmetic against the mirror's full checks, without a GPU."""
import pytest

from nnabla_b200 import functions as F

CASES = [
    ((2, 3, 10, 10), (4, 3, 3, 2), (0, 1), (1, 2), (2, 1), 1),
    ((1, 8, 7, 1), (8, 4, 7, 1), None, None, None, 2),
    ((5, 16, 9, 64), (32, 16, 5, 5), (2, 2), (2, 2), (1, 1), 1),
]


@pytest.mark.parametrize("x,w,pad,stride,dilation,group", CASES)
def test_convolution_geometry(monkeypatch, x, w, pad, stride, dilation, group):
    got = F.L.conv2d(x, w, None, 1, pad, stride, dilation, group)
    monkeypatch.setattr(F.L, "conv2d", lambda *a: None)
    assert got == F._conv_geometry(x, w, None, 1, pad, stride, dilation, group)


@pytest.mark.parametrize("x,w,pad,group", [((2, 3, 4, 4), (4, 3, 7, 7), (1, 1), 1), ((2, 3, 8, 8), (4, 2, 3, 3), None, 1),
                                           ((2, 4, 8, 8), (3, 2, 3, 3), None, 2), ((2, 4, 8), (3, 4, 3, 3), None, 1)])
def test_operands_that_do_not_fit_are_left_to_the_full_checks(x, w, pad, group):
    assert F.L.conv2d(x, w, None, 1, pad, None, None, group) is None
    with pytest.raises(RuntimeError):
        F._conv_geometry(x, w, None, 1, pad, None, None, group)
