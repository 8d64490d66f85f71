"""The binding's shape arithmetic against the mirror's full checks, without a GPU."""
import os
import re
import subprocess

import pytest
import torch

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


def test_the_callers_device_comes_back_on_every_way_out(tmp_path):
    """The binding changes the current device in one class only; that class, compiled against a stand-in for torch's two
    calls, puts the caller's device back after a block that ends and after one that throws."""
    text = open(os.path.join(os.path.dirname(F.__file__), "csrc", "native.cpp")).read()
    guard = re.search(r"^class OnDevice \{.*?^\};\n", text, re.S | re.M).group(0)
    assert re.search(r"set_?device\(", text.replace(guard, ""), re.I) is None
    source, program = tmp_path / "guard.cpp", tmp_path / "guard"
    source.write_text("""
#include <stdexcept>
namespace c10 {
using DeviceIndex = signed char;
namespace cuda {
int now = 2, changes = 0;
DeviceIndex current_device() { return (DeviceIndex)now; }
void set_device(DeviceIndex d) { now = d, ++changes; }
int SetDevice(DeviceIndex d) { return now = d, ++changes, 0; }
} // namespace cuda
} // namespace c10
%s
using namespace c10::cuda;
int main() {
  { const OnDevice on(2); if (now != 2 || changes != 0) return 1; }
  if (now != 2 || changes != 0) return 2;
  { const OnDevice on(5); if (now != 5) return 3; }
  if (now != 2 || changes != 2) return 4;
  try { const OnDevice on(7); throw std::runtime_error("out of memory"); } catch (const std::runtime_error &) {}
  return now == 2 ? 0 : 5;
}
""" % guard)
    subprocess.check_call([os.environ.get("CXX", "g++"), "-std=c++17", "-o", str(program), str(source)])
    assert subprocess.run([str(program)]).returncode == 0


@pytest.mark.parametrize("source,residual", [(-1, None), (1, None), (0, -1), (0, 1)])
def test_folded_convolutions_of_results_that_do_not_exist(source, residual):
    """No step reads a result that no step before it has: -1 is neither the last result nor no residual."""
    import types
    prepared = types.SimpleNamespace(side=torch.zeros(64, 576, dtype=torch.int8), group=1, shape=(64, 64, 3, 3))
    step = (source, prepared, torch.ones(64), None, (1, 1), (1, 1), residual, True, True)
    with pytest.raises(IndexError):
        F.folded_convolutions(torch.zeros(1, 64, 64, dtype=torch.int8), (1, 64, 8, 8), (step,), 2.0 ** -4)
