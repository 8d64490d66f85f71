"""Chains of dependent launches on two streams at once, from two threads: each gives the bits that it gives alone."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _folded(seed):
    from nnabla_b200 import functions as F
    from nnabla_b200 import resnet18
    params = resnet18.init_parameters(np.random.RandomState(seed), num_classes=16)
    net = resnet18.FoldedRunner(F, {k: torch.from_numpy(v).cuda() for k, v in params.items()})
    x = torch.randn(3, 3, 96, 96, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
    return lambda: [net(x)]


def _training(seed):
    """A binary-weight layer: convolution, batch statistics, gradients; tensor-core kernels in front of streaming ones."""
    from nnabla_b200 import functions as F
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w = r(8, 64, 20, 20), r(96, 64, 3, 3)
    wb, alpha, dy = torch.empty_like(w), torch.empty(96, device="cuda"), r(8, 96, 20, 20)
    beta, gamma = r(96), r(96)
    geometry = dict(pad=(1, 1))

    def step():
        y = F.binary_weight_convolution(x, w, wb, alpha, None, **geometry)
        z, mean, var = F.batch_normalization(y, beta, gamma, torch.zeros_like(beta), torch.ones_like(beta), output_stat=True)
        dy1, dbeta, dgamma = F.batch_normalization_backward(y, dy, gamma, mean, var)
        return [z, dbeta, dgamma, *F.binary_weight_convolution_backward(x, wb, alpha, dy1, **geometry)]
    return step


@pytest.mark.parametrize("first,second", [(_folded, _folded), (_folded, _training), (_training, _training)])
def test_two_streams(first, second):
    from nnabla_b200 import functions as F
    calls = [first(1), second(2)]
    want = [call() for call in calls]
    torch.cuda.synchronize()
    results, errors = [[], []], []

    def run(i):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(30):
                    results[i].append(calls[i]())
            stream.synchronize()
        except Exception as e:  # shown by the thread that waits
            errors.append(e)
    threads = [threading.Thread(target=run, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    F.check_device_status()
    for got, reference in zip(results, want):
        assert len(got) == 30
        for tensors in got:
            assert all(torch.equal(a, b) for a, b in zip(tensors, reference))
