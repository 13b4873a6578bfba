"""One network called with changing sizes, forward and training mixed: every call's outputs
and gradients are those of a network that has seen its size alone."""
from __future__ import annotations

import numpy as np
import pytest

from briefmatch_gb300 import learn

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no GPU", allow_module_level=True)

SIZES = [(2, 20, 30), (1, 24, 40), (2, 20, 30), (1, 5, 131)]


def _inputs(B, h, w):
    g = torch.Generator(device="cuda")
    g.manual_seed(B * 1000 + h * 10 + w)
    x = (torch.rand(B, h, w, 32, device="cuda", generator=g) * 2 - 1).to(torch.bfloat16)
    t = torch.rand(B, h, w, 3, device="cuda", generator=g)
    return x, t


def _call(net, size, train):
    B, h, w = size
    x, t = _inputs(*size)
    out = torch.empty(B, h, w, 3, device="cuda")
    grad = torch.zeros(net.nparam, device="cuda")
    torch.cuda.synchronize()
    net.set_input(x.data_ptr(), B, h, w)
    if train:
        net.train_step(B, h, w, t.data_ptr(), 0.0, grad.data_ptr())
    net.forward(B, h, w, out.data_ptr())
    torch.cuda.synchronize()
    net.check()
    return out.cpu().numpy(), grad.cpu().numpy()


@pytest.mark.parametrize("mode", [1, 2])
def test_alternating_sizes(mode):
    net = learn.load_net(learn.DEFAULT_WEIGHTS, 2, 24, 40)
    net.set_umma(mode)
    for k, (size, train) in enumerate([(s, t) for s in SIZES for t in (False, True)] + [(SIZES[1], False), (SIZES[0], True)]):
        alone = learn.load_net(learn.DEFAULT_WEIGHTS, 2, 24, 40)
        alone.set_umma(mode)
        want, got = _call(alone, size, train), _call(net, size, train)
        alone.close()
        assert np.array_equal(got[0], want[0]), k
        # (sums meet in the gradient in any order: a few of its own roundings apart)
        assert np.abs(got[1] - want[1]).max() <= 1e-5 * max(np.abs(want[1]).max(), 1e-30), k
    net.close()
