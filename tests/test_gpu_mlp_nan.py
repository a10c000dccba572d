"""A sample weight that is not a number makes the loss and every gradient not a number: the mean over the weights is."""
import math

import pytest
import torch

from dftbaby_b200 import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 130])
def test_weight_not_a_number(n):
    net = learned.GuessNet(device="cuda")
    g = torch.Generator(device="cuda").manual_seed(n)
    f, t = torch.randn(n, 8, device="cuda", generator=g), torch.rand(n, 2, device="cuda", generator=g)
    w = torch.ones(n, device="cuda")
    w[n // 2] = math.nan
    loss, grads = net.loss_and_gradients(f, t, w)
    assert math.isnan(loss)
    # biases of the output layer and of units that some sample switches on
    assert bool(torch.isnan(grads[5]).all()) and bool(torch.isnan(grads[4]).all())
    X = ((f - net.mean) / net.std).to(torch.bfloat16).float()
    H1 = torch.relu(X @ net.W1b[:, :8].float().T + net.b1).to(torch.bfloat16).float()
    H2 = torch.relu(H1 @ net.W2b.float().T + net.b2)
    on = (H2 > 1e-3).any(0)
    assert bool(on.any()) and bool(torch.isnan(grads[3][on]).all())
