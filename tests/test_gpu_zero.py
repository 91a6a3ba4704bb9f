"""Gradients start from zero: the flat buffer's memset, and two backward passes
in a row that do not add up."""
import numpy as np
import pytest
import torch

from mosaic_gb300 import _lib, engine
from mosaic_gb300.surrogate import MLP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 5, 1023, 1 << 20])
def test_zero(cuda, n):
    x = torch.full((n + 2,), 3.0, device=cuda)
    _lib.check(_lib.load().mk_zero(x.data_ptr() + 4, 4 * n, engine._stream_handle()))
    assert float(x[0]) == 3.0 and float(x[-1]) == 3.0 and not bool(x[1:n + 1].any())


@pytest.mark.parametrize("groups", [1, 2])
def test_gradients_do_not_add_up(cuda, groups):
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    lead = (groups,) if groups > 1 else ()
    net = MLP(8, 16, hidden=32, n_hidden=2, seed=1, groups=groups)
    X = torch.rand(lead + (40, 8), generator=g, device=cuda).bfloat16()
    T = torch.rand(lead + (40, 16), generator=g, device=cuda)

    def grads():
        acts, posts, Y = net.forward(X)
        _, G, Gb = net.mse(Y, T, torch.ones(16, device=cuda))
        dW, db = net.backward(acts, posts, G, Gb)
        return [x.clone() for x in list(dW) + list(db)]
    for a, b in zip(grads(), grads()):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-7)
